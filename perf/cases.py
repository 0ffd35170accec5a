"""Workloads of the KV-cache compression path, for timing and for comparing two builds.

Every case is one call (or one streaming step) that a user of the package makes through its
public entry points, on inputs as the path meets them:

* ``attn``    one attention call with column sums (``ops.attn_colsum`` on the cache layout, or
              ``ops.flash_attn_bias_colsum``, the drop-in call with a bias on every key);
* ``window``  one step of a sliding-window stream (``KVManager``: append, plain attention, prune);
* ``h2o``     one step of a heavy-hitter stream whose layers hand over the raw output of their QKV
              projection (``HeavyHittersKV.append_qkv``);
* ``stac``    one step of the full stream (``STACVoxelKV``: append and attend per layer, positions,
              retrieval on the streaming loop's schedule, prune = selection + merge + compaction);
* ``memory``  one insert into the voxel memory and one retrieval (``VoxelKVMerger``);
* ``points``  predicted point maps to voxel ids (``pointmap_to_positions``, ``BinaryVoxel``).

Queries and keys look like those of a trained layer after its q/k normalisation: rows of norm
sqrt(head_dim), a direction all queries share (some keys are heavy hitters, the scores of a head
spread over more than a decade), and keys of one image patch that resemble each other from frame
to frame (so that evicted tokens do merge into pivots).  World points come from a camera that
hovers in front of a depth surface, so the same voxels are seen again and again.
"""

import math

import torch

D = 64                   # head_dim of the path
SPECIAL = 5              # camera and register tokens in front of every frame's patches
VOXEL = 0.05
PATCH = 14
CYCLE = 8                # chunks of points that a stream's timed steps walk through
DEV = "cuda"


# ------------------------------------------------------------------------------------ cases
def listed():
    frame = dict(rows=37, cols=28)       # 518 x 392 images, patch 14: 1041 tokens a frame
    return [
        # one frame against a short cache: two frames' keys (the shortest of the attention benchmark's sweep)
        dict(name="attn_frame_short", kind="attn", m=1041, n=2082, pivots=0, heads=16, subsample=1.0, drop_in=False),
        # one frame against 32 frames of keys (the longest of that sweep)
        dict(name="attn_frame_long", kind="attn", m=1041, n=33312, pivots=0, heads=16, subsample=1.0, drop_in=False),
        # the drop-in operator: [T, H, D] tensors, a bias on every key, a quarter of the rows scored, ragged sizes
        dict(name="attn_drop_in_biased", kind="attn", m=2603, n=6247, pivots=0, heads=12, subsample=0.25, drop_in=True),
        # frame-by-frame streaming with the plain sliding window
        dict(name="window_frame", kind="window", layers=24, heads=16, chunk=1, window=8, **frame),
        # heavy-hitter streaming behind the fused projection epilogue, two frames at a time, 12 layers
        dict(name="h2o_fused_epilogue", kind="h2o", layers=12, heads=16, chunk=2, window=4, hh=2, subsample=1.0, **frame),
        # the smallest stream: toy model of two layers, small images; launches and host time are all of it
        dict(name="stac_small", kind="stac", layers=2, heads=4, chunk=2, window=4, hh=1, retrieval=1, subsample=1.0,
             rows=9, cols=7),
        # full model, frame by frame (lowest latency per frame)
        dict(name="stac_frame", kind="stac", layers=24, heads=16, chunk=1, window=4, hh=2, retrieval=2, subsample=1.0,
             **frame),
        # full model, chunks of four frames, window of eight: the headline stream
        dict(name="stac_chunk", kind="stac", layers=24, heads=16, chunk=4, window=8, hh=2, retrieval=2, subsample=1.0,
             **frame),
        # the same stream on one GPU of eight that share its heads
        dict(name="stac_head_shard", kind="stac", layers=24, heads=2, chunk=4, window=8, hh=2, retrieval=2, subsample=1.0,
             **frame),
        # voxel memory under pressure: 384 heads, eight frames evicted per call, pools bounded at 1 M slots
        dict(name="memory_bounded", kind="memory", heads=384, frames=8, dtype="bf16", slots=1_000_000, retrieve=2048,
             **frame),
        # one layer's voxel memory in fp32, unbounded
        dict(name="memory_fp32", kind="memory", heads=16, frames=8, dtype="fp32", slots=0, retrieve=2048, **frame),
        # a chunk's point maps to voxel ids
        dict(name="points_chunk", kind="points", frames=4, **frame),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "window", "h2o", "stac", "stac", "stac", "memory", "memory", "points"])
    if kind == "attn":
        m, n, heads = _log_int(rng, 64, 4164), _log_int(rng, 128, 33312), rng.choice([1, 2, 4, 8, 12, 16])
        n = min(n, max(128, 4164 * 17697 * 16 // (m * heads)))
        drop_in = rng.random() < 0.3
        pivots = 0 if drop_in or rng.random() < 0.4 else _log_int(rng, 16, min(4096, n - 64) if n > 128 else 32)
        return dict(kind="attn", m=m, n=n, pivots=pivots, heads=heads, subsample=rng.choice([1.0, 1.0, 0.5, 0.25]),
                    drop_in=drop_in)
    grid = dict(rows=_log_int(rng, 6, 37), cols=_log_int(rng, 5, 28))
    if kind == "memory":
        return dict(kind="memory", heads=_log_int(rng, 4, 256), frames=rng.randint(1, 8), dtype=rng.choice(["bf16", "bf16", "fp32"]),
                    slots=rng.choice([0, 0, 400_000]), retrieve=_log_int(rng, 64, 2048), **grid)
    if kind == "points":
        return dict(kind="points", frames=rng.randint(1, 16), **grid)
    layers, heads, chunk = _log_int(rng, 2, 24), rng.choice([2, 4, 6, 8, 12, 16]), rng.randint(1, 4)
    window = chunk * rng.randint(1, 2) + rng.randint(0, 3)
    case = dict(kind=kind, layers=layers, heads=heads, chunk=chunk, window=window, **grid)
    if kind != "window":
        case.update(hh=rng.randint(1, 2), subsample=rng.choice([1.0, 1.0, 0.5]))
    if kind == "stac":
        case.update(retrieval=rng.randint(1, 2))
    return case


# ------------------------------------------------------------------------------------ inputs
class _Source:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape):
        return torch.randn(*shape, device=DEV, generator=self.g)

    def uniform(self, *shape):
        return torch.rand(*shape, device=DEV, generator=self.g)

    def scores(self, *shape):
        """Heavy-hitter scores: positive, spread over decades."""
        return torch.exp(self.normal(*shape))


def _rows(x):
    """Rows of norm sqrt(D), bf16 (what a normalised query or key looks like)."""
    return (x * (math.sqrt(D) / x.norm(dim=-1, keepdim=True))).to(torch.bfloat16)


def _queries(src, u, tokens, *lead):
    """[*lead, tokens, H, D]: every query leans towards the head's shared direction u [H, D]."""
    return _rows(src.normal(*lead, tokens, u.shape[0], D) + 3.5 * u)


def _keys(src, u, tokens, frames, *lead):
    """[*lead, H, frames * tokens, D]: tokens of one patch resemble each other across frames, and lean
    towards the shared direction by an amount of their own."""
    H = u.shape[0]
    base = src.normal(*lead, H, 1, tokens, D) + 2.4 * src.normal(*lead, H, 1, tokens, 1) * u.view(H, 1, 1, D)
    base = base / base.norm(dim=-1, keepdim=True) * math.sqrt(D)
    noise = src.normal(*lead, H, frames, tokens, D)
    return _rows(base * math.sqrt(0.78) + noise * math.sqrt(0.22)).reshape(*lead, H, frames * tokens, D)


def _direction(src, heads):
    u = src.normal(heads, D)
    return u / u.norm(dim=-1, keepdim=True)


def _camera_points(src, frames, rows, cols, special=SPECIAL, dense=1):
    """World points [frames, special + rows * cols, 3] and mask: a camera that hovers (sines of
    incommensurate periods, millimetre jitter, slow drift) in front of a depth surface fixed in the
    world, depth 1 to 10 m; the special tokens are zero points with mask 0."""
    rows, cols = rows * dense, cols * dense
    y, x = torch.meshgrid((torch.arange(rows, device=DEV) + 0.5) / rows - 0.5,
                          (torch.arange(cols, device=DEV) + 0.5) / cols - 0.5, indexing="ij")
    x, y = (x * 1.2)[None], (y * 0.9)[None]
    amp, freq, phase = src.uniform(4), src.uniform(4, 2) * 3 + 0.5, src.uniform(4) * 2 * math.pi
    t = torch.arange(frames, device=DEV, dtype=torch.float32)
    jitter = src.normal(frames, 3) * 0.0005
    w = 2 * math.pi * t
    pos = torch.stack([0.08 * torch.sin(w / 97) + 0.0002 * t, 0.0125 * torch.sin(w / 53), 0.025 * torch.sin(w / 61)], 1) + jitter
    px, py, pz = (pos[:, i].view(-1, 1, 1) for i in range(3))
    depth = torch.full((frames, rows, cols), 5.0, device=DEV)
    for _ in range(3):
        wx, wy = x * depth + px, y * depth + py
        wave = sum(amp[i] * torch.sin(freq[i, 0] * wx * 0.5 + freq[i, 1] * wy * 0.5 + phase[i]) for i in range(4))
        depth = (5.5 + 4.5 * wave / amp.sum()).clamp(1.0, 10.0) - pz
    world = torch.stack([x * depth + px, y * depth + py, depth + pz], -1)
    if dense > 1:
        return world, src.uniform(frames, rows, cols) + 0.95
    pts = torch.zeros(frames, special + rows * cols, 3, device=DEV)
    mask = torch.zeros(frames, special + rows * cols, dtype=torch.bool, device=DEV)
    pts[:, special:] = world.reshape(frames, -1, 3)
    mask[:, special:] = src.uniform(frames, rows * cols) < 0.95
    return pts, mask


class _Rope:
    """Frequency tables of a 2-D rotary embedding, computed once per length (the interface that
    ``append_qkv`` expects of a layer's ``rope`` module)."""

    def __init__(self, base=100.0):
        self.base, self.cache = base, {}

    def _compute_frequency_components(self, dim, seq_len, device, dtype):
        key = (dim, seq_len, device, dtype)
        if key not in self.cache:
            inv = 1.0 / self.base ** (torch.arange(0, dim, 2, device=device).float() / dim)
            angles = torch.arange(seq_len, device=device).float()[:, None] * inv[None]
            angles = torch.cat([angles, angles], -1).to(dtype)
            self.cache[key] = (angles.cos().to(dtype), angles.sin().to(dtype))
        return self.cache[key]


def _tokens(case):
    return SPECIAL + case["rows"] * case["cols"]


# ------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    src = _Source(seed)
    return {"attn": _prepare_attn, "memory": _prepare_memory, "points": _prepare_points}.get(case["kind"], _prepare_stream)(case, src)


def _prepare_attn(case, src):
    M, N, P, H = case["m"], case["n"], case["pivots"], case["heads"]
    u = _direction(src, H)
    st = dict(case=case, q=_queries(src, u, M))
    k, v = _keys(src, u, N, 1), (src.normal(H, N, D) / 2).to(torch.bfloat16)
    if case["drop_in"]:
        counts = torch.floor(1 + 8 * src.uniform(H, N) ** 3)          # tokens that a key stands for
        st.update(q=st["q"][None], k=k.transpose(0, 1).contiguous()[None], v=v.transpose(0, 1).contiguous()[None],
                  bias=torch.log(counts)[None])
        return st
    hot = N - P
    st.update(k=k[:, :hot].contiguous(), v=v[:, :hot].contiguous(), hot=hot)
    if P:
        bias = torch.log(1 + 20 * src.uniform(H, P))
        live = (P * (0.75 + 0.25 * src.uniform(H, 1))).long()
        bias = torch.where(torch.arange(P, device=DEV)[None] < live, bias, torch.full_like(bias, -math.inf))
        st.update(kr=k[:, hot:].contiguous(), vr=v[:, hot:].contiguous(), br=bias)
    return st


def _manager(case):
    from stac_b200.stac import HeavyHittersKV, KVManager, STACVoxelKV
    kind, chunk, window, hh = case["kind"], case["chunk"], case["window"], case.get("hh", 0)
    kw = dict(num_layers=case["layers"], num_heads=case["heads"], head_dim=D, token_per_frame=_tokens(case),
              buffer_size=chunk + 1 + window + hh, chunk_size=chunk, recent_size=window, pinned_idx=[0],
              device=torch.device(DEV), dtype=torch.bfloat16)
    if kind == "window":
        kv = KVManager(**kw)
    else:
        kw.update(hh_size=hh, temperature=0.9, subsample_ratio=case["subsample"], attn_backend="cuda")
        if kind == "h2o":
            kv = HeavyHittersKV(**kw)
        else:
            share = case["layers"] * case["heads"] * 2_000_000 // 16       # 2 M slots per layer of 16 heads
            kv = STACVoxelKV(voxel_size=VOXEL, init_voxels=4096, voxel_buf_cap=8, voxel_piv_cap=4, voxel_backend="cuda",
                             sim_threshold=0.8, replace_threshold=0.8, score_threshold=0.2, slab_cap=10000, seg_size=1,
                             allocator="segment", retrieval_size=case["retrieval"], max_buffer_slots=share,
                             max_pivot_slots=share, **kw)
    kv.reset()
    return kv


def _stream_sets(case, src, u):
    """Two chunks' queries, keys and values per layer (behind the projection: its raw output), taken in turn."""
    L, H, chunk, tpf = case["layers"], case["heads"], case["chunk"], _tokens(case)
    T, sets = chunk * tpf, []
    for _ in range(2):
        q = _queries(src, u, T, L, 1)                                    # [L, 1, T, H, D]
        k = _keys(src, u, tpf, chunk, L, 1)                              # [L, 1, H, T, D]
        v = (src.normal(L, 1, H, T, D) / 2).to(torch.bfloat16)
        if case["kind"] == "h2o":
            kt, vt = (t.transpose(2, 3) for t in (k, v))
            sets.append(torch.stack([q, kt, vt], 3).reshape(L, 1, T, 3 * H * D))
        else:
            sets.append((q, k, v))
    return sets


def _chunks_seen(case):
    """Chunks that a stream has behind it when the timed steps begin."""
    live = 1 + case["window"] + case.get("hh", 0) + case["chunk"]
    return max(96 if case["kind"] == "stac" else 0, live + 2 * case["chunk"]) // case["chunk"]


def _retrieval_due(case, step):
    """The streaming loop's schedule in the steady state: once per window's worth of chunks."""
    return step % max(1, case["window"] // case["chunk"]) == 0


@torch.no_grad()
def _prepare_stream(case, src):
    """A stream in its steady state: the cache is full, the voxel memory holds what the frames seen so
    far have left in it, the retrieved pivots are in place.  The frames before the timed ones bring
    their heavy-hitter scores along instead of computing them."""
    kind, L, H, chunk, tpf = case["kind"], case["layers"], case["heads"], case["chunk"], _tokens(case)
    kv = _manager(case)
    T = chunk * tpf
    u = _direction(src, H)
    st = dict(case=case, kv=kv, step=0)
    if kind == "h2o":
        st["norms"] = [torch.nn.LayerNorm(D).to(DEV) for _ in range(2)]
        st["rope"] = _Rope()
        yx = torch.stack(torch.meshgrid(torch.arange(case["rows"], device=DEV), torch.arange(case["cols"], device=DEV),
                                        indexing="ij"), -1).reshape(-1, 2) + 1
        st["pos"] = torch.cat([torch.zeros(SPECIAL, 2, dtype=torch.int64, device=DEV), yx]).repeat(chunk, 1)[None]
    sets = _stream_sets(case, src, u)
    st["sets"] = sets
    seen = _chunks_seen(case)
    if kind == "stac":
        pts, mask = _camera_points(src, (seen + CYCLE) * chunk, case["rows"], case["cols"])
        pts, mask = pts.reshape(-1, T, 3), mask.reshape(-1, T)
        st["points"] = [(pts[i], mask[i]) for i in range(seen, seen + CYCLE)]
    for i in range(seen):
        x = sets[i % 2]
        for l in range(L):
            if kind == "h2o":
                kv.append_qkv(x[l], l, q_norm=st["norms"][0], k_norm=st["norms"][1], rope=st["rope"], pos=st["pos"])
            else:
                kv.append_kv(x[1][l], x[2][l], l)
        if kind != "window":
            live = kv.get_offset()[0]
            kv.get_scores()[:, :, :live].copy_(src.scores(L, H, live))
        if kind == "stac":
            kv.append_positions(pts[i], mask[i])
            if i == seen - 1:
                for l in range(L):
                    kv.retrieve_kv(l)
        kv.prune_kv()
    return st


@torch.no_grad()
def _prepare_memory(case, src):
    from stac_b200.stac.merger import VoxelKVMerger
    from stac_b200.stac.voxel import BinaryVoxel
    H, F, tpf = case["heads"], case["frames"], _tokens(case)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    vm = BinaryVoxel(voxel_size=VOXEL, device=DEV)
    pts, mask = _camera_points(src, 4 * F, case["rows"], case["cols"])
    pts, mask = pts.reshape(4, F * tpf, 3), mask.reshape(4, F * tpf)
    ids = [vm.upsert_points(pts[i], mask[i]) for i in range(4)]
    V = vm.get_voxel_num()
    bound = dict(max_buffer_slots=case["slots"], max_pivot_slots=case["slots"]) if case["slots"] else {}
    mem = VoxelKVMerger(H, D, init_voxels=V, pivot_cap=4, budget_cap=8, sim_thresh=0.8, replace_thresh=0.8,
                        score_thresh=0.2, dtype=dtype, device=torch.device(DEV), allocator="segment", seg_size=1, **bound)
    u = _direction(src, H)
    sets = []
    for i in range(2):
        K = _keys(src, u, tpf, F).to(dtype)
        Vv = (src.normal(H, F * tpf, D) / 2).to(dtype)
        vx = ids[i].view(1, -1).expand(H, -1).contiguous()
        around, count = vm.neighbor_ids(ids[i], 2)
        sets.append((K, Vv, src.scores(H, F * tpf), vx, around.clone(), count.clone()))
    for i in range(6):
        K, Vv, _, vx = sets[i % 2][:4]
        mem.insert_and_merge(K, Vv, src.scores(H, F * tpf), None, ids[i % 4].view(1, -1).expand(H, -1).contiguous(), V)
    return dict(case=case, mem=mem, sets=sets, voxels=V, step=0)


@torch.no_grad()
def _prepare_points(case, src):
    from stac_b200.stac.voxel import BinaryVoxel
    F = case["frames"]
    vm = BinaryVoxel(voxel_size=VOXEL, device=DEV)
    world, conf = _camera_points(src, CYCLE * F, case["rows"], case["cols"], dense=PATCH)
    maps = [(world[i * F:(i + 1) * F].contiguous(), conf[i * F:(i + 1) * F].contiguous()) for i in range(CYCLE)]
    return dict(case=case, vm=vm, maps=maps, step=0)


# ------------------------------------------------------------------------------------ run
def run(st):
    return {"attn": _run_attn, "memory": _run_memory, "points": _run_points}.get(st["case"]["kind"], _run_stream)(st)


def _run_attn(st):
    from stac_b200 import ops
    c = st["case"]
    if c["drop_in"]:
        return ops.flash_attn_bias_colsum(st["q"], st["k"], st["v"], bias=st["bias"], return_colsum=True,
                                          subsample_ratio=c["subsample"])
    return ops.attn_colsum(st["q"], st["k"], st["v"], st["hot"], st.get("kr"), st.get("vr"), st.get("br"), c["pivots"],
                           subsample_ratio=c["subsample"], want_lse=True)


@torch.no_grad()
def _run_stream(st):
    c, kv, step = st["case"], st["kv"], st["step"]
    kind, L = c["kind"], c["layers"]
    x = st["sets"][step % 2]
    layers = []
    for l in range(L):
        if kind == "h2o":
            q = kv.append_qkv(x[l], l, q_norm=st["norms"][0], k_norm=st["norms"][1], rope=st["rope"], pos=st["pos"])
        else:
            kv.append_kv(x[1][l], x[2][l], l)
            q = x[0][l]
        layers.append(kv.decode_sparse_attn(q, l))
    if kind == "stac":
        kv.append_positions(*st["points"][step % CYCLE])
        if _retrieval_due(c, step):
            for l in range(L):
                kv.retrieve_kv(l)
    kv.prune_kv()
    st["step"] = step + 1
    # every layer's output, and which tokens the cache holds now (global ids per layer and head)
    return {"layers": layers, "tokens": kv._token_indices_hot}


@torch.no_grad()
def _run_memory(st):
    K, V, S, vx, around, count = st["sets"][st["step"] % 2]
    st["step"] += 1
    st["mem"].insert_and_merge(K, V, S, None, vx, st["voxels"])
    return st["mem"].retrieve_device(around, count, st["case"]["retrieve"])


@torch.no_grad()
def _run_points(st):
    from stac_b200.stac.pointmap import pointmap_to_positions
    world, conf = st["maps"][st["step"] % CYCLE]
    st["step"] += 1
    pts, mask = pointmap_to_positions(world, conf, PATCH, conf_threshold=1.0, special_tokens_size=SPECIAL)
    return pts, mask, st["vm"].upsert_points(pts.view(-1, 3), mask.view(-1))


# ------------------------------------------------------------------------------------ work
def _scored_rows(m, ratio):
    """Query rows that the column sums run over (whole 128-row tiles)."""
    return m if ratio >= 1.0 else min(m, max(128, int(m * ratio) // 128 * 128))


def work(case):
    kind, H = case["kind"], case["heads"] if "heads" in case else 0
    if kind == "attn":
        M, N = case["m"], case["n"]
        r = _scored_rows(M, case["subsample"])
        return {"bytes": 4 * M * H * D + 4 * N * H * D + 4 * H * (M + N) + 4 * H * (N if case["drop_in"] else case["pivots"]),
                "flops": 4.0 * H * M * N * D + 2.0 * H * r * N * D}
    tpf = _tokens(case)
    if kind == "points":
        n = case["frames"] * case["rows"] * case["cols"]
        return {"bytes": n * 4 * 16 + case["frames"] * tpf * (12 + 1 + 4 + 8), "flops": n * 100.0}
    if kind == "memory":
        eb = 2 if case["dtype"] == "bf16" else 4
        E, R = H * case["frames"] * tpf, H * case["retrieve"]
        # new tokens in (K, V, score, voxel id) and into their segments; pivots out (K, V, mask, bias)
        return {"bytes": E * (4 * D * eb + 12) + R * (4 * D * eb + 5), "flops": 8.0 * E * D}
    # a stream's step, per (layer, head): new q, k, v in, output out, the cache and the pivots read once,
    # new tokens and their ids written; after the selection the kept tokens behind the first dropped one
    # change place (K, V, id, score, count) and the dropped ones go to the voxel memory
    LH, T = case["layers"] * H, case["chunk"] * tpf
    live = (1 + case["window"] + case.get("hh", 0) + case["chunk"]) * tpf
    keep, pivots = live - T, case.get("retrieval", 0) * tpf
    r = _scored_rows(T, case["subsample"]) if kind != "window" else 0
    per_head = T * (3 + 1 + 2) * 2 * D + 8 * T + (live + pivots) * 4 * D + (keep - tpf) * (4 * D + 16)
    if kind == "stac":
        per_head += T * (4 * D + 12) + pivots * 4 * D // max(1, case["window"] // case["chunk"])
    return {"bytes": LH * per_head, "flops": LH * (4.0 * T + 2.0 * r) * (live + pivots) * D}


def tolerance(case):
    kind = case["kind"]
    if kind == "points":
        return "exact"
    if kind == "memory":
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1e-5}
    if kind == "attn":
        return {"rel": 1e-2}
    # scores that differ in the last bits may swap two tokens of a row at the cut of the selection,
    # which moves the ids between them by one place
    return {"rel": 1e-2, "differ": 5e-3}


# ------------------------------------------------------------------------------------ exact
def _attention64(q, k, v, bias, rows, correction):
    """One head in 64 bits: q [M, D], k and v [N, D], bias [N] or None -> output, log-sum-exp, column sums over ``rows``."""
    s = q.double() @ k.double().T / math.sqrt(D)
    if bias is not None:
        s += bias.double()
    lse = torch.logsumexp(s, 1)
    p = torch.exp(s - lse[:, None])
    return p @ v.double(), lse, p[rows].sum(0) * correction


@torch.no_grad()
def exact(case, seed):
    """What the first pass returns, in 64 bits: the attention calls, and the sliding-window stream, whose cache
    holds the first frame and the last ``window`` ones whatever the scores are.  The other kinds build on
    the selections of all their earlier steps (``None``); the point maps are compared bit by bit."""
    src = _Source(seed)
    if case["kind"] == "attn":
        st = _prepare_attn(case, src)
        M, H = case["m"], case["heads"]
        r = _scored_rows(M, case["subsample"])
        rows = torch.arange(r, device=DEV) * (M // r)
        q = st["q"][0] if case["drop_in"] else st["q"]
        per_head = []
        for h in range(H):
            if case["drop_in"]:
                k, v, b = st["k"][0, :, h], st["v"][0, :, h], st["bias"][0, h]
            else:
                k, v, b = st["k"][h], st["v"][h], None
                if case["pivots"]:
                    k, v = torch.cat([k, st["kr"][h]]), torch.cat([v, st["vr"][h]])
                    b = torch.cat([torch.zeros(st["hot"], device=DEV), st["br"][h]])
            per_head.append(_attention64(q[:, h], k, v, b, rows, M / r))
        out, lse, colsum = (torch.stack([x[i] for x in per_head], 1 if i == 0 else 0) for i in range(3))
        return (out[None], lse[None], colsum[None]) if case["drop_in"] else (out, lse, colsum)
    if case["kind"] == "window":
        tpf, chunk, seen = _tokens(case), case["chunk"], _chunks_seen(case)
        sets = _stream_sets(case, src, _direction(src, case["heads"]))
        frames = [0] + list(range(seen * chunk - case["window"], (seen + 1) * chunk))
        where = [((f // chunk if f < seen * chunk else 0) % 2, f % chunk * tpf) for f in frames]
        layers = []
        for l in range(case["layers"]):
            k, v = (torch.cat([sets[i][j][l, 0, :, a:a + tpf] for i, a in where], 1) for j in (1, 2))
            q = sets[0][0][l, 0]
            layers.append(torch.stack([_attention64(q[:, h], k[h], v[h], None, slice(0, 0), 1.0)[0]
                                       for h in range(case["heads"])], 1)[None])
        return {"layers": layers, "tokens": None}
    return None
