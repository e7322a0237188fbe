"""Timed cases of the attention entry points: one dict of plain values per case.

Every case is one attention layer of a model: q, k, v lie on the GPU, one public call gives the output. Inputs come
from `spargeattn_b200.synthetic`: a smooth 3-D latent grid plus noise (video / image transformers; `t`, `h`, `w` is
the grid, `text` prompt tokens before it) or rotary-encoded noise with large sink keys (causal prefill, `t` = 0).

Keys of a case: entry (public function), B, H, N, D, dtype, layout, causal, t, h, w, text, and the selection:
  topk > 0    share of the key blocks that each query block visits
  cdf > 0     cumulative-probability threshold (around it per head where `tuned`)
  keep > 0    Bernoulli share of live blocks of a caller-made block mask
sim is the self-similarity below which a block is never left out, pv the P.V skip threshold (the entry points' default
50 never fires), sink keeps the first key block always.
"""
import math

import torch

import spargeattn_b200 as S
from spargeattn_b200 import synthetic

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
TOPK, CDF, MASK = "spas_sage2_attn_meansim_topk_cuda", "spas_sage2_attn_meansim_cuda", "block_sparse_sage2_attn_cuda"
TOPK_F16PV, CDF_F16PV = "spas_sage_attn_meansim_topk_cuda", "spas_sage_attn_meansim_cuda"


def _case(entry, B, H, D, dtype="bf16", layout="HND", grid=(0, 0, 0), text=0, N=None, causal=False, topk=0.0, cdf=0.0,
          keep=0.0, tuned=False, sim=-0.1, pv=50.0, sink=False, **name):
    t, h, w = grid
    return dict(entry=entry, B=B, H=H, N=N or text + t * h * w, D=D, dtype=dtype, layout=layout, causal=causal, t=t, h=h,
                w=w, text=text, topk=topk, cdf=cdf, keep=keep, tuned=tuned, sim=sim, pv=pv, sink=sink, **name)


def listed():
    return [
        # the smallest call of the repository's workloads: a few blocks per head, latency and launches count
        _case(TOPK, 1, 4, 64, grid=(8, 16, 16), topk=0.5, name="small_d64"),
        # a short causal prompt in the layout projections produce, batch of two, ragged length, fp16
        _case(TOPK, 2, 8, 128, "fp16", "NHD", N=1000, causal=True, topk=0.5, name="short_causal_nhd"),
        # one image of 64 x 64 latents behind 512 prompt tokens
        _case(TOPK, 1, 24, 128, grid=(1, 64, 64), text=512, topk=0.5, name="image_4608"),
        # cdf selection, ragged middle length, fp16
        _case(CDF, 1, 16, 128, "fp16", grid=(20, 20, 20), text=191, cdf=0.9, sim=0.1, name="cdf_8191"),
        # workload 1: both halves of a guidance batch, many small heads
        _case(TOPK, 2, 30, 64, grid=(13, 30, 45), text=226, topk=0.5, name="video_17776_d64"),
        # the same layer under a block mask that the caller made
        _case(MASK, 2, 30, 64, grid=(13, 30, 45), text=226, keep=0.4, name="block_mask_17776_d64"),
        # workload 2, the benchmark's default
        _case(TOPK, 1, 12, 128, grid=(21, 39, 40), topk=0.5, name="video_32760"),
        # the same layer as a tuned model calls it: thresholds per head, P.V skip test on
        _case(CDF, 1, 12, 128, grid=(21, 39, 40), cdf=0.8, sim=0.1, tuned=True, pv=5.0, name="tuned_32760"),
        # workload 3: long causal prefill, 32 heads
        _case(TOPK, 1, 32, 128, N=32768, causal=True, topk=0.5, name="prefill_32768"),
        # workload 4: the largest layer
        _case(TOPK, 1, 24, 128, grid=(33, 45, 80), text=256, topk=0.4, name="video_119056"),
        # fp16 P.V entry point at the benchmark's shape, fp16 tensors
        _case(TOPK_F16PV, 1, 12, 128, "fp16", grid=(21, 39, 40), topk=0.5, name="f16pv_32760"),
        # fp16 P.V with cdf selection: causal prefill with small heads, token-major layout, bf16
        _case(CDF_F16PV, 1, 16, 64, layout="NHD", N=8192, causal=True, cdf=0.8, name="f16pv_causal_cdf_8192_d64"),
    ]


LARGEST = 24 * 119056.0 ** 2 * 128 * 0.4        # B H N^2 D times the share of live blocks


def draw(rng):
    """Another layer: lengths from 256 to 119 056 and 1 to 64 heads over their logarithm, every entry point."""
    while True:
        entry = rng.choice([TOPK, TOPK, TOPK, CDF, CDF, MASK, TOPK_F16PV, CDF_F16PV])
        B, H = rng.choice([1, 1, 1, 2, 3]), round(math.exp(rng.uniform(0, math.log(40))))
        N = round(math.exp(rng.uniform(math.log(256), math.log(119056))))
        c = _case(entry, B, H, rng.choice([64, 128, 128]), rng.choice(["bf16", "bf16", "fp16"]), rng.choice(["HND", "HND", "NHD"]),
                  N=N, causal=entry != MASK and rng.random() < 0.3)
        if not c["causal"]:
            c["t"] = rng.randint(1, max(1, min(33, N // 128)))
            c["h"] = max(1, int(math.sqrt(N / c["t"] * rng.uniform(0.5, 1.0))))
            c["w"] = max(1, N // (c["t"] * c["h"]))
            c["text"] = N - c["t"] * c["h"] * c["w"]
        if entry in (TOPK, TOPK_F16PV):
            c["topk"] = round(rng.uniform(0.2, 0.7), 2)
        elif entry == MASK:
            c["keep"] = round(rng.uniform(0.2, 0.7), 2)
        else:
            c["cdf"], c["tuned"] = round(rng.uniform(0.6, 0.95), 3), rng.random() < 0.5
            c["sim"] = -0.1 if c["causal"] else 0.1
        c["pv"] = rng.choice([50.0, 50.0, 50.0, 5.0, 15.0])
        c["sink"] = rng.random() < 0.2
        if B * H <= 64 and B * H * float(N) ** 2 * c["D"] * _share(c) <= LARGEST and B * H * N * c["D"] <= 24 * 119056 * 128:
            return c


def prepare(case, seed):
    B, H, N, D, dtype = case["B"], case["H"], case["N"], case["D"], DTYPES[case["dtype"]]
    gen = torch.Generator("cuda").manual_seed(seed)
    if case["t"] == 0:
        q, k, v = synthetic.llm_prefill_qkv(B, H, N, D, seed, "cuda", dtype)
    else:
        q, k, v = (torch.empty(B, H, N, D, dtype=dtype, device="cuda") for _ in range(3))
        for i in range(B * H):                    # head by head: the generator's fp32 intermediates are large
            one = synthetic.video_qkv(1, 1, (case["t"], case["h"], case["w"]), D, seed * 4096 + i, "cuda", case["text"], True, dtype)
            for all_heads, head in zip((q, k, v), one):
                all_heads[i // H, i % H] = head[0, 0]
    if case["layout"] == "NHD":
        q, k, v = (x.transpose(1, 2).contiguous() for x in (q, k, v))
    kw = {"tensor_layout": case["layout"], "pvthreshd": case["pv"], "attention_sink": case["sink"]}
    if case["entry"] == MASK:
        kw["mask_id"] = synthetic.bernoulli_block_mask(B, H, N, case["keep"], seed, "cuda")
    else:
        kw["is_causal"] = case["causal"]
        if case["topk"]:
            kw["topk"] = case["topk"]
        if case["cdf"]:
            kw["cdfthreshd"] = case["cdf"]
        kw["simthreshd1"] = case["sim"]
    if case["tuned"]:                             # what a tuned model keeps: thresholds found for each head
        spread = lambda lo, hi: lo + (hi - lo) * torch.rand(H, generator=gen, device="cuda")
        kw["cdfthreshd"] = spread(case["cdf"] - 0.02, case["cdf"] + 0.02)
        kw["simthreshd1"] = spread(case["sim"] - 0.1, case["sim"] + 0.02)
        kw["pvthreshd"] = spread(case["pv"], case["pv"] + 5.0)
    return getattr(S, case["entry"]), q, k, v, kw


def run(state):
    fn, q, k, v, kw = state
    return fn(q, k, v, **kw)


def _share(case):
    """Share of the N x N score blocks that the selection keeps (cdf: about what these inputs give)."""
    if case["cdf"]:
        return case["cdf"] / 2 if case["causal"] else case["cdf"] ** 2
    live = case["topk"] or case["keep"]
    return live - live * live / 2 if case["causal"] else live


def work(case):
    """q, k, v and a mask read once, the output written once; the two products of every live 128 x 64 block."""
    B, H, N, D = case["B"], case["H"], case["N"], case["D"]
    nq, nk = (N + 127) // 128, (N + 63) // 64
    blocks = B * H * nq * nk
    return {"bytes": 4 * 2 * B * H * N * D + (4 * blocks if case["keep"] else 0),
            "flops": 4.0 * D * 128 * 64 * blocks * _share(case)}


def tolerance(case):
    """FP8 P.V: a probability keeps three mantissa bits (rms rounding error 2.6 %), and an implementation that meets the
    blocks in another order rounds against another running maximum; over the keys of a row that leaves up to 2 % of the
    output. fp16 P.V: the rounding of the 16-bit output."""
    if case["entry"] in (TOPK_F16PV, CDF_F16PV):
        return {"rel": 5e-3 if case["dtype"] == "bf16" else 2e-3}
    return {"rel": 2e-2}
