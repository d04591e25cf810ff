"""What the speed of this framework is measured on: one pass of each thing that a long-video generator has it do.

A generator calls the package in a handful of ways, and every kind of case below is one of them:

* `attend`   -- the HSA layer itself: a chunk of queries over the key/value window (`HSAAttention`).  Called once per
  block and denoising step, so it is most of what the package does.
* `write`    -- what comes before it in every block: RMSNorm + rotary embedding of q and k, and the chunk's rows and
  compressed slots written into the layer caches (`rope.qk_norm_rope`, `HSAAttention.append_kv`).
* `generate` -- the chunk loop around both (`ChunkPipeline.generate`): denoising forwards and one clean-context forward
  per chunk, launched call by call.
* `store`    -- a prompt switch, first half: the populated window goes into the HKV bank (`HKVCache.store`).
* `install`  -- second half: pages are retrieved and installed into the online cache, and the compressed tier is
  rebuilt (`HKVCache.retrieve`, `HKVCache.apply`); from HBM, or from page-locked host memory, which is the default tier.
* `gather`   -- per-head page retrieval with nothing on the host: scores and top-k for all layers, copy records built on
  the device, one page-copy launch per 65535 records.

Sizes are those of the repository's benchmark configurations (12 heads of 128, frames of 1560 tokens, windows of 21
frames, chunks of 3, histories of 480 frames) and, in `draw`, everything between them and the smallest calls of the tests.
"""
import math

import torch

from worldattention_b200 import hsa_stage, rope
from worldattention_b200.causal_dit import CausalDiT, ChunkPipeline, DiTConfig, rope_table
from worldattention_b200.hkv import HKVCache, temporal_band, temporal_complex_dims
from worldattention_b200.hkv.install import build_records_device, gather_records_device
from worldattention_b200.hkv.retrieval import score_and_topk_layers
from worldattention_b200.hsa import HSAAttention

DEV = torch.device("cuda", 0)
D = 128                                   # head_dim of every configuration of this repository
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp32": 4}
# Share of the key blocks that cumulative-mass routing keeps on the inputs below, measured; it only enters `work`.
MASS_SHARE = 0.33
TEXT_TOKENS, TEXT_DIM = 512, 4096


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def listed():
    window = dict(kind="attend", batch=1, heads=12, frame=1560, q_frames=3, kv_frames=21, dtype="bf16", coarse=True)
    return [
        # The smallest calls: a one-frame chunk of a small latent at the start of a rollout, default class options, no
        # compressed cache yet.  Latency and launches.
        dict(window, name="attend small", frame=390, q_frames=1, kv_frames=3, block=64, routing="mass", coarse=False),
        # float32 layer, one latent frame over three: the accuracy configuration (default class options).
        dict(window, name="attend fp32", q_frames=1, kv_frames=3, block=64, routing="mass", dtype="fp32", coarse=False),
        # First chunk of a rollout: the window holds the chunk itself.
        dict(window, name="attend first chunk", kv_frames=3, block=128, routing="mass"),
        # Steady state, fixed head-adaptive block counts: the headline configuration.
        dict(window, name="attend window", block=128, routing="topk"),
        # Steady state with the class's defaults: 64-token blocks and counts from the cumulative mass.
        dict(window, name="attend window mass", block=64, routing="mass"),
        # A history of 480 frames kept in the cache (748 800 tokens).
        dict(window, name="attend long history", kv_frames=480, block=64, routing="topk"),
        # The chunk's tokens prepared and written into a layer's caches.
        dict(name="write chunk", kind="write", heads=12, frame=1560, frames=3, window=21, block=128),
        # Seven chunks of generation through a model of four blocks, from an empty window to a full one.
        dict(name="generate", kind="generate", layers=4, heads=12, frame_h=30, frame_w=52, window=21, chunks=7, block=128),
        # A full window of a 30-block model goes into the bank's HBM tier.
        dict(name="store window", kind="store", layers=30, heads=12, frame=1560, frames=21, page_frames=3),
        # Four pages of three frames come back, from the HBM tier for 30 blocks ...
        dict(name="install hot", kind="install", layers=30, heads=12, frame=1560, window=21, page_frames=3, topk=4, banked=2, hot=True),
        # ... and from page-locked host memory (the default tier) for four.
        dict(name="install host", kind="install", layers=4, heads=12, frame=1560, window=21, page_frames=3, topk=4, banked=2, hot=False),
        # Sixteen of 480 pages per head and layer, gathered on the device.
        dict(name="gather per head", kind="gather", layers=30, heads=12, frame=1560, pages=480, resident=64, topk=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; half of them are attention calls, as in use."""
    kind = rng.choice(["attend"] * 5 + ["write", "generate", "store", "install", "gather"])
    heads = rng.choice([8, 12, 12, 12, 16, 24])
    frame = _log_int(rng, 150, 1560)                     # tokens of a latent frame, any number
    if kind == "attend":
        dtype = rng.choice(["bf16"] * 5 + ["fp32"])
        q_frames = rng.randint(1, 3)
        most = 24 if dtype == "bf16" else 6
        if dtype == "bf16" and rng.random() < 0.25:
            most = 240
        kv_frames = q_frames + _log_int(rng, 1, most) - 1
        return dict(kind=kind, batch=rng.choice([1, 1, 1, 2]) if kv_frames <= 24 else 1, heads=heads if dtype == "bf16" else 12,
                    frame=frame, q_frames=q_frames, kv_frames=kv_frames, block=rng.choice([64, 128]),
                    routing=rng.choice(["mass", "topk"]) if kv_frames <= 24 else "topk", dtype=dtype, coarse=rng.random() < 0.75)
    if kind == "write":
        frames = rng.randint(1, 3)
        return dict(kind=kind, heads=rng.choice([8, 12, 16]), frame=frame, frames=frames, window=frames + _log_int(rng, 1, 30),
                    block=rng.choice([64, 128]))
    if kind == "generate":
        chunks = rng.randint(2, 5)
        return dict(kind=kind, layers=rng.randint(1, 4), heads=12, frame_h=rng.randint(8, 30), frame_w=rng.randint(12, 52),
                    window=3 * chunks, chunks=chunks, block=rng.choice([64, 128]))
    if kind == "store":
        return dict(kind=kind, layers=rng.randint(4, 30), heads=12, frame=frame, frames=rng.randint(3, 21), page_frames=rng.randint(1, 8))
    if kind == "install":
        return dict(kind=kind, layers=rng.randint(4, 30), heads=12, frame=frame, window=rng.randint(12, 21),
                    page_frames=rng.randint(1, 4), topk=rng.randint(1, 6), banked=rng.randint(1, 3), hot=True)
    return dict(kind=kind, layers=rng.randint(2, 30), heads=12, frame=frame, pages=_log_int(rng, 40, 960), resident=40,
                topk=rng.randint(2, 24))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _tokens(g, batch, n, heads, dtype, spread=0.0):
    """`[batch, n, heads, D]`: unit normal values plus, with `spread`, an offset shared by 130 neighbouring tokens (a patch
    of the picture), so that blocks of keys differ from one another as they do in a video."""
    x = torch.empty((batch, n, heads, D), dtype=dtype, device=DEV)
    step = 130 * 512
    for s in range(0, n, step):
        m = min(step, n - s)
        part = torch.randn((batch, m, heads, D), generator=g, device=DEV)
        if spread:
            off = torch.randn((batch, -(-m // 130), heads, D), generator=g, device=DEV) * spread
            part += off.repeat_interleave(130, dim=1)[:, :m]
        x[:, s:s + m] = part
    return x


def _hsa(g, heads, block, frame, dtype=None):
    """An HSA layer with weights as after training has moved them off their block-average start."""
    hsa = HSAAttention(heads, D, block_size=block, proj_segment_len=frame)
    hsa_stage.init_hsa_parameters(hsa)
    hsa = hsa.to(DEV)
    with torch.no_grad():
        for p in (hsa.k_proj_mat, hsa.v_proj_mat):
            p.add_((torch.randn(p.shape, generator=g, device=DEV) * (0.3 / block)).to(p.dtype))
        hsa.gate_lin.weight.copy_(torch.randn((D, D), generator=g, device=DEV) * 0.05)
        hsa.gate_lin.bias.copy_(torch.randn((D,), generator=g, device=DEV) * 0.2)
    return hsa if dtype is None else hsa.to(dtype)


def _topk(g, heads, block, kv_blocks):
    counts = torch.tensor([4, 8, 16, 32], device=DEV)[torch.randint(0, 4, (heads,), generator=g, device=DEV)]
    if kv_blocks > 2048:                                  # a long history: the same budget for every head
        counts = torch.full((heads,), 16, device=DEV)
    return (counts * (128 // block)).clamp(max=kv_blocks).to(torch.int32)


def _prepare_attend(c, seed):
    g, dtype = _gen(seed), DTYPES[c["dtype"]]
    lq, lkv = c["q_frames"] * c["frame"], c["kv_frames"] * c["frame"]
    hsa = _hsa(g, c["heads"], c["block"], c["frame"])
    if c["routing"] == "topk":
        hsa.topk_per_head = _topk(g, c["heads"], c["block"], -(-lkv // c["block"]))
    s = {"hsa": hsa, "q": _tokens(g, c["batch"], lq, c["heads"], dtype, 1.0), "k": _tokens(g, c["batch"], lkv, c["heads"], dtype, 1.0),
         "v": _tokens(g, c["batch"], lkv, c["heads"], dtype), "kc": None, "vc": None}
    if c["coarse"]:
        s["kc"], s["vc"] = hsa.compress_kv_cache(s["k"], s["v"])
    return s


def _run_attend(s):
    with torch.no_grad():
        return s["hsa"](s["q"], s["k"], s["v"], k_coarse=s["kc"], v_coarse=s["vc"])


def _prepare_write(c, seed):
    g, h, frame = _gen(seed), c["heads"], c["frame"]
    n, size = c["frames"] * frame, c["window"] * frame
    hsa = _hsa(g, h, c["block"], frame, torch.bfloat16)
    table = torch.view_as_real(rope_table(D)).to(DEV).contiguous()
    coarse = hsa.coarse_cache_size(size)
    weights = [(1 + 0.1 * torch.randn((h * D,), generator=g, device=DEV)).to(torch.bfloat16) for _ in range(2)]
    width = next(w for w in range(int(math.isqrt(frame)), 0, -1) if frame % w == 0)
    return {"hsa": hsa, "table": table, "grid": (c["frames"], frame // width, width), "heads": h, "position": size - n,
            "start": c["window"] - c["frames"], "wq": weights[0], "wk": weights[1],
            "xq": _tokens(g, 1, n, h, torch.bfloat16).view(1, n, h * D), "xk": _tokens(g, 1, n, h, torch.bfloat16).view(1, n, h * D),
            "v": _tokens(g, 1, n, h, torch.bfloat16), "k_cache": _tokens(g, 1, size, h, torch.bfloat16),
            "v_cache": _tokens(g, 1, size, h, torch.bfloat16), "kc": _tokens(g, 1, coarse, h, torch.bfloat16),
            "vc": _tokens(g, 1, coarse, h, torch.bfloat16)}


def _run_write(s):
    with torch.no_grad():
        q = rope.qk_norm_rope(s["xq"], s["wq"], 1e-6, s["grid"], None, s["start"], heads=s["heads"], table=s["table"])
        k = rope.qk_norm_rope(s["xk"], s["wk"], 1e-6, s["grid"], None, s["start"], heads=s["heads"], table=s["table"])
        s["hsa"].append_kv(k, s["v"], s["k_cache"], s["v_cache"], s["kc"], s["vc"], position=s["position"])
    return {"q": q, "k": s["k_cache"], "v": s["v_cache"], "kc": s["kc"], "vc": s["vc"]}


def _prepare_generate(c, seed):
    g = _gen(seed)
    heads = c["heads"]
    blocks = -(-c["window"] * c["frame_h"] * c["frame_w"] // c["block"])
    cfg = DiTConfig(layers=c["layers"], heads=heads, dim=heads * D, latent_hw=(2 * c["frame_h"], 2 * c["frame_w"]),
                    window_frames=c["window"], hsa_block=c["block"], hsa_topk=_topk(g, heads, c["block"], blocks).tolist())
    with torch.random.fork_rng(devices=[0]), torch.device(DEV):
        torch.manual_seed(seed)
        model = CausalDiT(cfg)
    model.freqs = model.freqs.cpu()                       # the rotary table stays on the host, as the class keeps it
    model = model.to(DEV, torch.bfloat16).eval()
    model.init_hsa(seed)
    noise = torch.randn((1, c["chunks"] * cfg.frames_per_chunk, cfg.in_channels) + cfg.latent_hw, generator=g, device=DEV)
    return {"pipe": ChunkPipeline(model, device=DEV), "noise": noise.to(torch.bfloat16), "seed": seed,
            "prompt": torch.randn((TEXT_TOKENS, TEXT_DIM), generator=g, device=DEV).to(torch.bfloat16)}


def _run_generate(s):
    s["pipe"].reset(keep_buffers=True)                    # a new video
    latents = s["pipe"].generate(s["noise"], [s["prompt"]], generator=_gen(s["seed"]))
    return {"latents": latents, "caches": [[c[n] for n in ("k", "v", "k_coarse", "v_coarse")] for c in s["pipe"].kv_cache]}


def _online_cache(g, layers, heads, frame, frames, filled, hsa=None):
    """Per-layer caches as views of one tensor per name, and those tensors."""
    size = frames * frame
    slabs = {n: torch.empty((layers, 1, size, heads, D), dtype=torch.bfloat16, device=DEV) for n in ("k", "v")}
    if hsa is not None:
        slabs.update({n: torch.zeros((layers, 1, hsa.coarse_cache_size(size), heads, D), dtype=torch.bfloat16, device=DEV)
                      for n in ("k_coarse", "v_coarse")})
    for n in ("k", "v"):
        for layer in range(layers):
            slabs[n][layer].normal_(generator=g)
    slabs["k"][0] += _tokens(g, 1, size, heads, torch.bfloat16, 0.5) * 0.5      # layer 0 is what pages are indexed by
    cache = [{**{n: t[layer] for n, t in slabs.items()},
              "global_end_index": torch.full((1,), filled, dtype=torch.long, device=DEV),
              "local_end_index": torch.full((1,), filled, dtype=torch.long, device=DEV)} for layer in range(layers)]
    return cache, slabs


def _prompt(g):
    return torch.randn((1, TEXT_TOKENS, TEXT_DIM), generator=g, device=DEV).to(torch.bfloat16)


def _band():
    return temporal_band(rope_table(D), D).to(DEV)


def _prepare_store(c, seed):
    g = _gen(seed)
    cache, _ = _online_cache(g, c["layers"], c["heads"], c["frame"], c["frames"], c["frames"] * c["frame"])
    hkv = HKVCache(frame_seq_length=c["frame"], page_size_frames=c["page_frames"], topk_pages=4, hbm_max_chunks=2)
    return {"hkv": hkv, "cache": cache, "prompt": _prompt(g), "band": _band(), "frame": 2 * c["frames"]}


def _run_store(s):
    hkv = s["hkv"]
    hkv.reset()                                           # a new rollout; its first prompt switch
    chunk = hkv.store(s["cache"], prompt_embeds=s["prompt"], current_start_frame=s["frame"], temporal_freqs=s["band"])
    blob = hkv.tier.get(chunk)
    return {"chunk": chunk, "k": blob["k"], "v": blob["v"], "pages": hkv.chunks[chunk]["page_index"], "prompt": hkv.prompt_bank[chunk]}


def _prepare_install(c, seed):
    g = _gen(seed)
    hsa = [_hsa(g, c["heads"], 128, c["frame"], torch.bfloat16) for _ in range(c["layers"])]
    hkv = HKVCache(frame_seq_length=c["frame"], page_size_frames=c["page_frames"], topk_pages=c["topk"],
                   stage1_topk_chunks=min(2, c["banked"]), hbm_max_chunks=c["banked"] if c["hot"] else 0)
    size = c["window"] * c["frame"]
    for i in range(c["banked"]):
        cache, slabs = _online_cache(g, c["layers"], c["heads"], c["frame"], c["window"], size, hsa[0])
        prompt = _prompt(g)
        hkv.store(cache, prompt_embeds=prompt, current_start_frame=(i + 1) * c["window"], temporal_freqs=_band())
    torch.cuda.synchronize()                              # copies to the host tier have landed long before a later switch
    query = torch.randn((c["heads"] * D,), generator=g, device=DEV)
    return {"hkv": hkv, "cache": cache, "slabs": slabs, "hsa": hsa, "prompt": prompt, "query": query, "band": _band(),
            "frame": (c["banked"] + 1) * c["window"]}


def _run_install(s):
    hkv = s["hkv"]
    pages = hkv.retrieve(prompt_embeds=s["prompt"], query_vec=s["query"])
    tokens = hkv.apply(s["cache"], pages, current_start_frame=s["frame"], temporal_freqs=s["band"], hsa_modules=s["hsa"])
    return {"pages": pages, "tokens": tokens, **s["slabs"]}


def _prepare_gather(c, seed):
    g = _gen(seed)
    layers, heads, frame, resident = c["layers"], c["heads"], c["frame"], min(c["resident"], c["pages"])
    pool = torch.empty((2, layers, resident, frame, heads, D), dtype=torch.bfloat16, device=DEV)
    for i in range(2):
        for layer in range(layers):
            pool[i, layer].normal_(generator=g)
    page_bytes = frame * heads * D * 2
    slot = torch.randperm(c["pages"], generator=g, device=DEV) % resident       # which resident page stands for each id
    rot = torch.randn((c["topk"], temporal_complex_dims(D), 2), generator=g, device=DEV)
    return {"pool": pool, "src": [pool[i].data_ptr() + slot * page_bytes for i in range(2)], "topk": c["topk"], "heads": heads,
            "frame": frame, "layer_bytes": resident * page_bytes, "page_bytes": page_bytes,
            "index": torch.randn((layers, c["pages"], heads * D), generator=g, device=DEV) * 0.5,
            "query": torch.randn((heads * D,), generator=g, device=DEV),
            "rot": (rot / rot.norm(dim=-1, keepdim=True)).contiguous(),
            "cache": torch.zeros((2, layers, c["topk"] * frame, heads, D), dtype=torch.bfloat16, device=DEV)}


def _run_gather(s):
    row = s["heads"] * D
    scores, ids, vals = score_and_topk_layers(s["query"], s["index"], s["topk"], groups=s["heads"])
    records = torch.cat([build_records_device(ids, s["src"][i], dst=s["cache"][i], rotate=i == 0, src_layer_stride=s["layer_bytes"],
                                              src_token_stride=row, dst_layer_stride=s["topk"] * s["page_bytes"], dst_token_stride=row,
                                              page_tokens=s["frame"], head_dim=D) for i in range(2)])
    gather_records_device(records, max_tokens=s["frame"], row_elems=D, head_dim=D, dtype=torch.bfloat16, rotations=s["rot"],
                          n_temporal=temporal_complex_dims(D))
    return {"scores": scores, "ids": ids, "vals": vals, "cache": s["cache"]}


_PREPARE = {"attend": _prepare_attend, "write": _prepare_write, "generate": _prepare_generate, "store": _prepare_store,
            "install": _prepare_install, "gather": _prepare_gather}
_RUN = {"attend": _run_attend, "write": _run_write, "generate": _run_generate, "store": _run_store, "install": _run_install,
        "gather": _run_gather}


def prepare(case, seed):
    """The user's side of a call: inputs from the seed, weights and handles kept."""
    return _RUN[case["kind"]], _PREPARE[case["kind"]](case, seed)


def run(state):
    fn, s = state
    return fn(s)


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far correct results may lie apart
# ------------------------------------------------------------------------------------------------
def _work_attend(batch, heads, lq, lkv, lc, block, routing, size, rank_flops=0.0):
    blocks = -(-lkv // block)
    share = MASS_SHARE if routing == "mass" else min(1.0, (16 if blocks > 2048 else 15) * (128 / block) / blocks)
    row = batch * heads * D
    touched = 1 - (1 - share) ** (-(-lq // block))         # part of V that some query block selects
    read = row * (lq + lkv + touched * lkv + 2 * lc) * size + row * lq * size
    flops = 4.0 * row * lq * (share * lkv + lc) + 2.0 * row * lq * D + rank_flops
    return {"bytes": read, "flops": flops}


def work(case):
    c = case
    row = c["heads"] * D
    if c["kind"] == "attend":
        lq, lkv, rank = c["q_frames"] * c["frame"], c["kv_frames"] * c["frame"], -(-c["frame"] // c["block"])
        lc = c["kv_frames"] * rank
        w = _work_attend(c["batch"], c["heads"], lq, lkv, lc, c["block"], c["routing"], SIZE[c["dtype"]])
        if not c["coarse"]:                                # compressed here: all of V, and the projections
            w["flops"] += 4.0 * c["batch"] * row * lkv * rank
        return w
    if c["kind"] == "write":
        n, rank = c["frames"] * c["frame"], -(-c["frame"] // c["block"])
        # q in and out; k in, into the cache; v in, into the cache; the compressed slots
        return {"bytes": 2.0 * row * (6 * n + 2 * c["frames"] * rank), "flops": 4.0 * row * n * rank + 16.0 * row * n}
    if c["kind"] == "generate":
        frame, lq, rank = c["frame_h"] * c["frame_w"], 3 * c["frame_h"] * c["frame_w"], -(-c["frame_h"] * c["frame_w"] // c["block"])
        ffn, passes = 8960, 5
        linear = 2.0 * lq * row * (6 * row + 2 * ffn) + 4.0 * lq * TEXT_TOKENS * row    # q k v o, q o, FFN; text attention
        flops = nbytes = 0.0
        for i in range(c["chunks"]):
            frames = min(3 * (i + 1), c["window"])
            a = _work_attend(1, c["heads"], lq, frames * frame, frames * rank, c["block"], "topk", 2)
            flops += passes * c["layers"] * (linear + a["flops"])
            nbytes += passes * c["layers"] * (a["bytes"] + 2.0 * row * (6 * row + 2 * ffn))
        return {"bytes": nbytes, "flops": flops}
    if c["kind"] == "store":
        pages = -(-c["frames"] // c["page_frames"])
        return {"bytes": 2.0 * row * c["frames"] * c["frame"] * 4 * c["layers"] + 4.0 * pages * row, "flops": 8.0 * row * c["frames"] * c["frame"]}
    if c["kind"] == "install":
        pages = -(-c["window"] // c["page_frames"]) * min(2, c["banked"])
        frames = min(c["window"], c["page_frames"] * min(c["topk"], pages))
        rank = -(-c["frame"] // 128)
        # pages read, the whole cache written (the tail is cleared), the compressed tier written
        return {"bytes": 2.0 * 2 * row * c["layers"] * (frames * c["frame"] + c["window"] * (c["frame"] + rank)) + 4.0 * pages * row,
                "flops": 4.0 * row * c["layers"] * frames * c["frame"] * rank}
    moved = 2.0 * 2 * 2 * row * c["layers"] * min(c["topk"], c["pages"]) * c["frame"]     # K and V, read and written
    return {"bytes": moved + 4.0 * row * c["layers"] * c["pages"], "flops": 2.0 * row * c["layers"] * c["pages"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "attend":
        # bf16 products and a bf16 result; in float32 the sparse branch is still rounded to bf16 on its way in and out
        return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 2e-2}
    if kind == "write":
        return {"rel": 4e-3, "max": 2e-2}                  # one bf16 rounding per value
    if kind == "generate":
        return {"rel": 2e-2}                               # a chain of bf16 forwards, each fed with the one before
    if kind == "install":
        return {"rel": 4e-3, "max": 2e-2}                  # copies, one rotation rounded to bf16, one bf16 compression
    return {"rel": 1e-6, "max": 1e-5}                      # copies, and float32 sums and scores
