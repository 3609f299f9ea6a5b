"""Performance cases: the work a user has this framework do, through its public entry points.

Three kinds, each with its own ranges in draw():

  request   one sequence on a speculative engine: the prompt goes in, then tokens are generated (MTP drafter or prompt
            lookup, k drafts a cycle; k = 0 is plain decoding).  Prompts of 128 tokens and more take the dense prompt
            path, as the benchmark's do
  streams   several sequences on one engine: the prompts go in together, then cycles until every stream has its tokens
  gemm      the dequant-fused GEMM operator alone: f32 rows in, f32 rows out

Models are the benchmark's shapes (packs.cfg_c0, _c2, _c3, _c4) with seeded random weights.  A program loads a model
once and keeps it, so the engines of a model share one copy of the weights and a state owns its sequence only.
"""
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("eureka-engine_b200")
llb, packs = pkg.llb, pkg.packs

DENSE_PROMPT = 128       # prompts from this length on take the dense prompt path
GEMM_FMTS = ("Q4_K", "Q5_K", "Q6_K", "Q8_0")


def listed():
    return [
        # the operator's smallest call: one row against a small matrix, latency and launches only
        dict(name="gemm-small", kind="gemm", fmt="Q8_0", rows=1024, mats=1, cols=1024, T=1),
        # the largest matrices of a verify step, 27B shape: gate and up in one launch, four rows (k = 3)
        dict(name="gemm-gate-up", kind="gemm", fmt="Q4_K", rows=17408, mats=2, cols=5120, T=4),
        # a row count that fills no tile, the six-bit format of down projections, seven rows (two n-tiles)
        dict(name="gemm-ragged", kind="gemm", fmt="Q6_K", rows=5003, mats=1, cols=17408, T=7),
        # a chat turn on the small hybrid: short prompt, drafts partly accepted
        dict(name="chat-0.8b", kind="request", model="c0", k=3, prompt=64, new=48, sample=False),
        # the headline: 27B shape, MTP k = 3, batch 1
        dict(name="chat-27b", kind="request", model="c2", k=3, prompt=48, new=24, sample=False),
        # the same model without speculation: one row a pass
        dict(name="plain-27b", kind="request", model="c2", k=0, prompt=33, new=24, sample=False),
        # the headline's prompt: time to the first tokens of a long document
        dict(name="prompt-27b", kind="request", model="c2", k=3, prompt=3011, new=4, sample=False),
        # long context on the Q8_0 model, five drafts (six rows a pass)
        dict(name="long-9b", kind="request", model="c4", k=5, prompt=4096, new=24, sample=False),
        # sampled decoding (temperature, top-k, penalties) with one draft
        dict(name="sampled-9b", kind="request", model="c4", k=1, prompt=200, new=32, sample=True),
        # routed experts, prompt-lookup drafter, one user
        dict(name="chat-moe", kind="request", model="c3", k=3, prompt=96, new=32, sample=False),
        # routed experts, eight users of plain decoding on one copy of the weights
        dict(name="streams-moe", kind="streams", model="c3", k=0, streams=8, prompt=40, new=16),
        # four users with drafts: sixteen rows a pass
        dict(name="streams-27b", kind="streams", model="c2", k=3, streams=4, prompt=40, new=10),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["request"] * 5 + ["streams"] * 2 + ["gemm"] * 3)
    if kind == "gemm":
        cols = 256 * _log(rng, 4, 68)
        return dict(kind="gemm", fmt=rng.choice(GEMM_FMTS), rows=_log(rng, 512, 20000), mats=rng.choice([1, 1, 2]), cols=cols, T=rng.randint(1, 8))
    if kind == "streams":
        k, streams = rng.choice([(0, 2), (0, 8), (0, 16), (1, 4), (1, 8), (3, 2), (3, 4)])
        return dict(kind="streams", model=rng.choice(["c0", "c2", "c3", "c4"]), k=k, streams=streams, prompt=_log(rng, 9, 60), new=rng.randint(5, 12))
    model = rng.choice(["c0", "c2", "c3", "c4"])
    most = 150 if model == "c3" else 3000
    return dict(kind="request", model=model, k=rng.choice([0, 1, 3, 3, 5]), prompt=_log(rng, 12, most), new=rng.randint(8, 32),
                sample=rng.random() < 0.2)


# ---- models ---------------------------------------------------------------------------------------
def _cfg(model):
    if model == "c0":      # a gain at which some drafts are accepted and some are not
        return packs.cfg_c0(mix_gain=0.1)
    if model == "c3":      # a tied head and a small gain: the output comes back to earlier tokens, which prompt lookup needs
        return packs.cfg_c3(tied_head=True, mix_gain=0.07, type_overrides=(("token_embd", "Q6_K"),))
    return {"c2": packs.cfg_c2, "c4": packs.cfg_c4}[model]()


@functools.lru_cache(maxsize=None)
def _loaded(model, drafter):
    """The model's weights on the GPU, as an engine that the states' own engines share them with."""
    llb.init(torch.cuda.current_device())
    cfg = _cfg(model)
    pack = packs.build_pack(cfg, device="cuda")
    mtp = None
    if drafter and not cfg.n_experts:
        mtp = packs.aux1_bytes(packs.build_mtp(pack, draft_vocab=min(cfg.vocab_size, 40960), eh="embed" if model == "c0" else "hidden"))
    torch.cuda.synchronize()
    eng = llb.SpecEngine(pack, mtp, k=3 if drafter else 0, max_ctx=64)
    del pack
    torch.cuda.empty_cache()
    return eng


# ---- states ---------------------------------------------------------------------------------------
def _prompts(case, seed, vocab):
    """The prompt, or the streams' prompts of different lengths."""
    n, B = case["prompt"], case.get("streams", 1)
    return [packs.synth_prompt(1000003 * seed + b, max(2, n - b * n // (2 * B)), vocab) for b in range(B)]


def _weights(fmt, rows, cols, gen):
    """Device-layout weights of one matrix, drawn N(0, 0.02) and quantised."""
    raw = packs.QUANT[fmt](torch.randn(rows, cols, device="cuda", generator=gen) * 0.02).contiguous()
    w = torch.empty(llb.lib().llb_b200_weight_bytes(packs.FMT[fmt], rows, cols), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    llb.check(llb.lib().llb_b200_weight_upload(packs.FMT[fmt], rows, cols, raw.data_ptr(), 1, w.data_ptr()), "weight_upload")
    llb.check(llb.lib().llb_b200_sync(), "sync")
    return w


class _Planes:
    """The operator's activation handle, freed with the state."""

    def __init__(self, cols, T):
        self.h = llb.handle(llb.lib().llb_b200_xp_new(cols, T, 2), "xp_new")

    def __del__(self):
        llb.lib().llb_b200_xp_free(self.h)


def prepare(case, seed):
    if case["kind"] == "gemm":
        llb.init(torch.cuda.current_device())
        gen = torch.Generator(device="cuda").manual_seed(seed)
        w = [_weights(case["fmt"], case["rows"], case["cols"], gen) for _ in range(case["mats"])]
        x = torch.randn(case["T"], case["cols"], device="cuda", generator=gen)
        y = [torch.zeros(case["T"], case["rows"], device="cuda") for _ in w]
        torch.cuda.synchronize()
        return dict(case=case, w=w, x=x, y=y, xp=_Planes(case["cols"], case["T"]))
    prompts = _prompts(case, seed, _cfg(case["model"]).vocab_size)
    ctx = case["prompt"] + (case["new"] + 4) * (case["k"] + 1) + 32
    eng = _loaded(case["model"], case["k"] > 0).sibling(k=case["k"], max_ctx=ctx, streams=case.get("streams", 1))
    eng.set_prefill(case["prompt"] >= DENSE_PROMPT)
    if case.get("sample"):
        eng.set_sampler(llb.SmpParams.make(temp=0.8, top_p=0.95, top_k=40, repeat_penalty=1.1, seed=seed))
    return dict(case=case, eng=eng, prompts=prompts)


# ---- one pass -------------------------------------------------------------------------------------
def _words(ids, top2):
    """Emitted ids and the two largest logits of their rows."""
    return {"ids": np.asarray(ids, np.int32), "logits": np.ascontiguousarray(np.asarray(top2, np.uint32)[:, 1::2]).view(np.float32)}


def run(state):
    case = state["case"]
    if case["kind"] == "gemm":
        xp, w, y = state["xp"].h, state["w"], state["y"]
        llb.check(llb.lib().llb_b200_xp_set_f32(xp, state["x"].data_ptr()), "xp_set")
        llb.gemm(packs.FMT[case["fmt"]], [t.data_ptr() for t in w], [case["rows"]] * len(w), [t.data_ptr() for t in y], case["cols"], xp)
        return y
    eng, new = state["eng"], case["new"]
    if case["kind"] == "request":
        eng.prefill(state["prompts"][0])
        return _words(*eng.generate(new))
    eng.prefill_streams(state["prompts"])
    ids = [[] for _ in state["prompts"]]
    top2 = [[] for _ in state["prompts"]]
    while min(len(i) for i in ids) < new:
        for b, (i, t) in enumerate(eng.cycle_streams()):
            ids[b].extend(i)
            top2[b].extend(t)
    return _words(np.concatenate([i[:new] for i in ids]), np.concatenate([t[:new] for t in top2]))


# ---- what a pass cannot do without ----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sizes(model, drafter):
    """(bytes and multiply-adds of the weights a row meets, bytes of one routed expert and their number, the same of a
    draft, cache bytes of a position), all layers together."""
    cfg = _cfg(model)
    dense = expert = macs = draft = 0
    last = max(i for i in range(cfg.n_layers) if cfg.is_full(i))
    for name, rows, cols in packs.tensor_plan(cfg):
        ty = packs.tensor_type(cfg, name)
        nb = rows * (cols * 4 if ty == "F32" else packs.row_bytes(ty, cols))
        if "_exps." in name:
            expert += nb / cfg.n_experts
            macs += rows * cols / cfg.n_experts * cfg.n_experts_used
        elif name != "token_embd.weight" or cfg.tied_head:
            dense += nb
            macs += rows * cols
        if drafter and not cfg.n_experts and name.startswith("blk.%d." % last):
            draft += nb
    full = sum(1 for i in range(cfg.n_layers) if cfg.is_full(i))
    return dense, macs, expert, draft, full * 2 * cfg.n_kv_heads * cfg.head_dim * 4


def work(case):
    if case["kind"] == "gemm":
        ty, R, K, T = case["fmt"], case["rows"] * case["mats"], case["cols"], case["T"]
        return {"bytes": R * packs.row_bytes(ty, K) + 4 * T * (K + R), "flops": 2 * R * K * T}
    cfg = _cfg(case["model"])
    dense, macs, expert, draft, kv = _sizes(case["model"], case["k"] > 0)
    B, k, n, new = case.get("streams", 1), case["k"], case["prompt"], case["new"]
    # drafts are right often enough for k + 1 tokens a pass on c0 and c3 at best; on the other two they never are
    passes = -(-new // (k + 1)) if case["model"] in ("c0", "c3") else new
    rows = B * (k + 1 if not cfg.n_experts else 1)
    touched = min(cfg.n_experts, rows * cfg.n_experts_used) if cfg.n_experts else 0
    touched_prompt = min(cfg.n_experts, B * n * cfg.n_experts_used) if cfg.n_experts else 0
    by = passes * (dense + touched * expert + k * draft + B * kv * (n + new / 2)) + dense + touched_prompt * expert + B * kv * n
    return {"bytes": by, "flops": 2 * macs * (B * n + passes * rows)}


def tolerance(case):
    if case["kind"] == "gemm":      # f32 sums of f32 values that the operator keeps to about 22 bits
        return {"rel": 1e-5}
    # ids are whole numbers; the logits come through up to 64 layers that amplify the rounding of f32 sums
    return {"rel": 1e-3, "max": 1e-2, "differ": 0.01}
