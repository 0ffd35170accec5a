"""CPU-side checks: the C ABI library loads and exports every declared symbol, the product
refuses to run without a GPU (no CPU fallback), bench helpers, and the multi-rank timing logic
on two gloo ranks."""

import os
import re
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "stac_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(stac_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    import __graft_entry__
    __graft_entry__.build()
    from stac_b200 import _lib
    import ctypes
    names = _declared_functions()
    assert len(names) >= 15
    handle = ctypes.CDLL(_lib.LIB_PATH)
    for n in names:
        assert hasattr(handle, n), f"{n} declared in include/stac_b200.h but not exported"
        assert n in _lib.SIGNATURES, f"{n} has no ctypes signature"
    assert set(_lib.SIGNATURES) == set(names)
    lib = _lib.lib()
    assert lib.stac_abi_version() == 2
    assert lib.stac_status_string(1) == b"bad argument"
    # row log-sum-exps (+ 512 words of flags and counters, rounded up to 256 bytes) + two partial forward
    # results and two partial column-sum groups (3 x 128 keys) per CTA
    lse_bytes = ((1041 * 16 + 512) * 4 + 255) // 256 * 256
    assert lib.stac_attn_workspace_bytes(1041, 16) == lse_bytes + 2 * 160 * (128 * 64 + 2 * 128 + 3 * 128) * 4
    assert lib.stac_merge_scratch_bytes(4, 100, 1000) > 0
    assert lib.stac_voxel_scratch_bytes(10) == (10 + 16) * 8 + 16   # keys, key list padded to 16, counter


def test_every_thread_waits_for_the_kernel_before():
    """Kernels that may start while the one before them drains see what it and its predecessors wrote only in threads that have waited:
    no condition stands in front of a wait, and every kernel that is launched that way has one."""
    csrc = os.path.join(ROOT, "stac_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        text = open(os.path.join(csrc, name)).read()
        kernels = re.split(r"\n__global__ ", re.sub(r"//[^\n]*", "", text))[1:]
        for line in "\n".join(kernels).splitlines():
            assert "grid_dep_wait()" not in line or line.strip() == "grid_dep_wait();", (name, line)
        waiting = {re.search(r"(\w+_kernel)\s*\(", k).group(1): "  grid_dep_wait();" in k for k in kernels if re.search(r"(\w+_kernel)\s*\(", k)}
        for launched in re.findall(r"launch(?:_clusters)?_behind\([^;]*?(\w+_kernel)\b", text):
            assert waiting.get(launched, True), (name, launched)


def _plan(M, H, T_hot, T_ret, n_sm=148, workspace=1):
    import ctypes
    from stac_b200 import _lib
    parts, cluster = ctypes.c_int(-1), ctypes.c_int(-1)
    grid = _lib.lib().stac_attn_forward_plan(M, H, T_hot, T_ret, n_sm, workspace, ctypes.byref(parts), ctypes.byref(cluster))
    return grid, parts.value, cluster.value


def test_forward_plan():
    """In how many parts items are cut follows from the sizes (there is no device here to ask); the shapes of the attention tests take
    the paths that they are there for; every part has at least one tile and a CTA of one wave."""
    assert _plan(130, 3, 300, 0) == (6, 1, 0) and _plan(1041, 16, 2082, 0) == (144, 1, 0) and _plan(2600, 16, 800, 150) == (148, 1, 0)
    for shape, parts, cluster in [((64, 1, 12 * 112, 0), 4, 1), ((130, 3, 150, 6000), 8, 1), ((128, 1, 40000, 0), 20, 0), ((257, 6, 9000, 100), 6, 1),
                                  ((1100, 2, 2000, 100), 5, 1), ((700, 8, 2000, 0), 3, 0), ((4164, 2, 17697, 0), 2, 1), ((4164, 2, 3000, 300), 2, 1), ((128, 2, 40000, 0), 20, 0)]:
        items = (shape[0] + 127) // 128 * shape[1]
        assert _plan(*shape) == (parts * items, parts, cluster), (shape, _plan(*shape))
    assert _plan(128, 1, 40000, 0, workspace=0)[1:] == (8, 1)       # nowhere to leave more parts
    assert _plan(0, 1, 5, 0)[0] == 0 and _plan(1, 1, 0, 0)[0] == 0
    rs = np.random.RandomState(0)
    for _ in range(3000):
        M, H, T_hot, T_ret = (int(np.exp(rs.uniform(0, np.log(n)))) for n in (4200, 16, 40000, 4000))
        T_ret *= int(rs.randint(2))
        grid, parts, cluster = _plan(M, H, T_hot, T_ret)
        items, tiles = (M + 127) // 128 * H, -(-T_hot // 112) + -(-T_ret // 112)
        assert 1 <= parts <= tiles and (parts == 1 or (grid == parts * items <= 148)) and (not cluster or 2 <= parts <= 8)
        assert parts > 1 or grid == items or (grid == 148 <= items and tiles >= 8)


def test_struct_layout_matches_header():
    import ctypes
    from stac_b200 import _lib
    # 10 4-byte fields, 6 pointers + int (+pad), 7 pointers + int (+pad), 10 pointers, int (+pad), 2 pointers
    assert ctypes.sizeof(_lib.StacPool) == 40 + 6 * 8 + 8 + 7 * 8 + 8 + 10 * 8 + 8 + 8 + 8
    assert ctypes.sizeof(_lib.StacEvicted) == 8 * 8 + 8


def test_product_has_no_cpu_path():
    import torch
    from stac_b200 import _lib
    from stac_b200.stac import STACVoxelKV
    if torch.cuda.is_available():
        pytest.skip("GPU present")
    with pytest.raises(_lib.StacError):
        STACVoxelKV(num_layers=1, num_heads=2, head_dim=64, token_per_frame=8, buffer_size=4,
                    device=torch.device("cpu"), dtype=torch.bfloat16)
    import stac_b200.stac.stac_voxel as sv
    src = open(sv.__file__).read() + open(os.path.join(ROOT, "stac_b200", "ops.py")).read()
    assert "oracle" not in src


def test_manager_rejects_unsupported_config():
    import torch
    from stac_b200.stac.merger import VoxelKVMerger
    with pytest.raises(ValueError):
        VoxelKVMerger(4, 64, budget_cap=32, dtype=torch.bfloat16, device="cpu")
    with pytest.raises(ValueError):
        VoxelKVMerger(4, 128, budget_cap=8, dtype=torch.bfloat16, device="cpu")


def test_bench_helpers():
    sys.path.insert(0, ROOT)
    import bench
    pts = bench.synth_points(3, seed=1)
    pts2 = bench.synth_points(3, seed=1)
    tpf, ck = bench.CFG["tpf"], bench.CFG["chunk"]
    assert pts[0][0].shape == (ck * tpf, 3) and pts[0][1].shape == (ck * tpf,)
    assert all(np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) for a, b in zip(pts, pts2))
    assert not pts[0][1][:5].any() and not pts[0][1][tpf:tpf + 5].any()     # special tokens masked
    z = pts[1][0][pts[1][1]]
    assert np.isfinite(z).all()
    due = [i for i in range(12) if bench.retrieval_due(i)]
    assert due == [5, 7, 9, 11]
    assert bench.attn_flops(1041, 10376) == 6 * 16 * 1041 * 10376 * 64
    assert bench.job_throughput(32, 1000.0, 8) == 256.0


def test_cpu_arms_of_the_bench_step(monkeypatch):
    """The two CPU legs of bench.py (`cpu_baseline`, `--impl reference`): one chunk of one layer and
    one head through the numpy port and, where its sources are staged, through the reference's
    own manager; the record says what was measured and how it is scaled."""
    sys.path.insert(0, ROOT)
    import bench
    monkeypatch.setattr(bench, "CPU_SAMPLE", (1, 1))
    arms = [bench.PortCpuStream(1, 1)]
    if bench._reference_available():
        arms.append(bench.ReferenceCpuStream(1, 1))
    for st in arms:
        dt = st.step() + st.step()
        assert dt > 0.0
        rec = bench._cpu_record(st, dt, 2)
        assert rec["kind"] == st.kind and rec["scale_factor"] == 384.0 and rec["sample_rows"] == 1
        assert rec["value"] == round(bench.CFG["chunk"] * 2 / (dt * 384.0), 5)
        assert rec["cores"] >= 1 and "scaled x384" in rec["sample"]


def _rank_main(rank, world, port, q):
    import torch
    import torch.distributed as dist
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port), RANK=str(rank), WORLD_SIZE=str(world))
    dist.init_process_group("gloo", rank=rank, world_size=world)
    sys.path.insert(0, ROOT)
    import bench
    dist.barrier()
    ms = bench.max_over_ranks(100.0 + 50.0 * rank)
    q.put((rank, ms, bench.job_throughput(16, ms, world)))
    dist.barrier()
    dist.destroy_process_group()


def test_two_rank_timing_is_max_over_ranks():
    """world_size 2 on gloo: each rank streams independently; the job time is the slower rank's."""
    import torch.multiprocessing as mp
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = 29500 + os.getpid() % 1000
    procs = [ctx.Process(target=_rank_main, args=(r, 2, port, q)) for r in range(2)]
    for p in procs:
        p.start()
    res = sorted(q.get(timeout=120) for _ in range(2))
    for p in procs:
        p.join(timeout=60)
        assert p.exitcode == 0
    assert [r[1] for r in res] == [150.0, 150.0]
    assert all(abs(r[2] - 32 / 0.15) < 1e-9 for r in res)


def _shard_rank_main(rank, world, port, q):
    import torch
    import torch.distributed as dist
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port), RANK=str(rank), WORLD_SIZE=str(world))
    dist.init_process_group("gloo", rank=rank, world_size=world)
    sys.path.insert(0, ROOT)
    from stac_b200.sharding import gather_head_counts, head_slice
    L, H = 3, 8
    full = torch.arange(L * H, dtype=torch.int32).reshape(L, H) * 7 % 11
    sl = head_slice(rank, world, H)
    got = gather_head_counts(full[:, sl].reshape(-1), L)
    q.put((rank, got.tolist(), full.tolist(), [sl.start, sl.stop]))
    dist.barrier()
    dist.destroy_process_group()


def test_head_sharding_counts_two_ranks():
    """Head-sharded stream: every rank ends with the per-head retrieval counts of all heads."""
    import torch.multiprocessing as mp
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = 29600 + os.getpid() % 1000
    procs = [ctx.Process(target=_shard_rank_main, args=(r, 2, port, q)) for r in range(2)]
    for p in procs:
        p.start()
    res = sorted(q.get(timeout=120) for _ in range(2))
    for p in procs:
        p.join(timeout=60)
        assert p.exitcode == 0
    assert res[0][3] == [0, 4] and res[1][3] == [4, 8]
    for _, got, full, _ in res:
        assert got == full
    from stac_b200.sharding import head_slice
    with pytest.raises(ValueError):
        head_slice(0, 3, 16)


def test_launch_state_is_kept_per_device(tmp_path):
    """The shared-memory opt-in of a kernel and the SM count belong to a GPU: the bookkeeping the
    launchers use (csrc/per_device.h, host-only C++) keeps one entry per device ordinal."""
    import subprocess
    src = tmp_path / "per_device_test.cpp"
    src.write_text('#include "per_device.h"\n'
                   "int main() {\n"
                   "  stac::PerDeviceFlag f;\n"
                   "  stac::PerDeviceValue<int> sm;\n"
                   "  if (!f.needs_setup(0) || !f.needs_setup(1)) return 1;\n"
                   "  f.mark(0);\n"
                   "  if (f.needs_setup(0)) return 2;\n"
                   "  if (!f.needs_setup(1)) return 3;          // device 1 still has to opt in\n"
                   "  sm.set(0, 148);\n"
                   "  if (sm.get(0) != 148 || sm.get(1) != 0) return 4;\n"
                   "  if (!stac::device_index_ok(63) || stac::device_index_ok(64) || stac::device_index_ok(-1)) return 5;\n"
                   "  return 0;\n"
                   "}\n")
    exe = tmp_path / "per_device_test"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "stac_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0
    # no launcher keeps a process-wide "attribute already set" or SM-count static any more
    for name in ("attn_colsum.cu", "h2o.cu", "retrieve.cu", "voxel.cu"):
        text = open(os.path.join(ROOT, "stac_b200", "csrc", name)).read()
        assert not re.search(r"static\s+(bool|int)\s+(attr_done|attr_smem|n_sm)\b", text), name


def test_checkpoint_file_loads_without_pickle(tmp_path):
    """save_state / load_state round trip of a state dictionary with every value type the managers
    emit (tensors, lists, numbers, strings, None, nested dicts), read back with weights_only=True."""
    import torch
    from stac_b200.stac.checkpoint import load_state, save_state

    class Stub:
        device = torch.device("cpu")

        def __init__(self):
            self.loaded = None

        def state_dict(self):
            return {"format": 1, "class": "STACVoxelKV", "shape": [2, 3, 64, 21, 147], "use_cpu": False,
                    "key": torch.arange(12, dtype=torch.bfloat16).view(2, 3, 2), "key_cpu": None,
                    "offset_hot": [5, 5], "temperature": 0.9,
                    "memory": {"meta": torch.arange(8, dtype=torch.int32), "over": {"S": torch.zeros(0)},
                               "voxel_alloc": 64},
                    "retrieved": [torch.ones(2, 2), torch.zeros(2, dtype=torch.bool)]}

        def load_state_dict(self, sd):
            self.loaded = sd

    a, b = Stub(), Stub()
    path = str(tmp_path / "stream.pt")
    save_state(a, path)
    load_state(b, path)
    want = a.state_dict()
    assert b.loaded["offset_hot"] == want["offset_hot"] and b.loaded["key_cpu"] is None
    assert torch.equal(b.loaded["key"], want["key"]) and b.loaded["key"].dtype == torch.bfloat16
    assert torch.equal(b.loaded["memory"]["meta"], want["memory"]["meta"])
    assert b.loaded["retrieved"][1].dtype == torch.bool


def test_no_grad_wrapper_restores_the_mode():
    """Gradients are off inside, whatever they were before is restored, also when the function raises."""
    import torch
    from stac_b200._lib import no_grad

    @no_grad
    def inside(fail=False):
        if fail:
            raise KeyError("x")
        return torch.is_grad_enabled()
    for before in (True, False):
        with torch.set_grad_enabled(before):
            assert inside() is False and torch.is_grad_enabled() is before
            try:
                inside(fail=True)
            except KeyError:
                pass
            assert torch.is_grad_enabled() is before


def test_running_scores_are_checked_before_their_pointers_are_used():
    """Rows that overlap are refused by the C entry, and tensors that do not hold what the kernel writes by the caller."""
    import torch
    from stac_b200 import _lib, ops
    H, M, T = 2, 128, 300
    need = _lib.lib().stac_attn_workspace_bytes(M, H)
    p = 1 << 20                                   # aligned; nothing is read before the arguments are checked

    def call(stride):
        return _lib.lib().stac_attn_colsum_scored(p, H * 64, p, p, 64, T * 64, T, None, None, 64, 64, 0, None, 0, p, H * 64,
                                                  None, p, T, M, H, 64, 0.125, 1.0, p, p, stride, 0, M, 0.9, p, need,
                                                  None, None)
    assert call(T - 1) == 1 and call(0) == 1      # STAC_ERR_BAD_ARG
    dev = torch.device("cpu")
    good = torch.zeros(H, T + 5)
    ops._check_score_update(good, good.clone(), T + 5, H, T, dev)
    ops._check_score_update(good[:, :T], good[:, :T], T + 5, H, T, dev)
    bad = [good.double(), good.half(), good.to("meta"), good[:1], good[:, :T - 1], good.t().contiguous().t(),
           torch.zeros(1, T + 5).expand(H, T + 5), good.flatten()]
    for t in bad:
        for pair in ((t, good), (good, t)):
            with pytest.raises(AssertionError):
                ops._check_score_update(*pair, T + 5, H, T, dev)
    with pytest.raises(AssertionError):
        ops._check_score_update(good, good, T, H, T, dev)


def test_captured_calls_have_a_workspace_of_their_own(monkeypatch):
    """The workspace kept for eager calls of a stream is not handed to a call that is captured on it (the
    graph would outlive it, and would run beside eager calls), nor one of a capture to an eager call."""
    import torch
    from stac_b200 import ops

    dev = torch.device("cpu")
    capturing = [False]
    monkeypatch.setattr(ops, "stream_ptr", lambda device=None: 7)
    monkeypatch.setattr(ops, "_workspaces", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    eager = ops._attn_workspace(dev, 8, 2)
    assert ops._attn_workspace(dev, 8, 2) is eager
    capturing[0] = True
    a, b = ops._attn_workspace(dev, 8, 2), ops._attn_workspace(dev, 8, 2)
    assert a is not eager and b is not eager and a is not b
    assert all(int(t[:ops.ATTN_CTL_WORDS].count_nonzero()) == 0 for t in (a, b))
    capturing[0] = False
    assert ops._attn_workspace(dev, 8, 2) is eager


@pytest.mark.parametrize("without,code", [
    ("import sys; sys.modules['torch'] = None", "import stac_b200._lib as l; assert l.lib().stac_abi_version() == 2"),
    ("import torch; del torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice",
     """
import stac_b200._lib as l, stac_b200.ops, stac_b200.stac as s
for use in (l.stream_ptr, lambda: s.KVManager(num_layers=1, num_heads=2, head_dim=64, token_per_frame=8, buffer_size=4,
                                              device="cpu", dtype=torch.bfloat16)):
    try:
        use()
    except l.StacError:
        continue
    raise SystemExit("no StacError")
"""),
], ids=["no torch", "torch without CUDA"])
def test_import_needs_no_cuda_build_of_torch(without, code):
    """The ctypes binding loads without torch; with a torch that was built without CUDA the package imports
    and says so at the first use."""
    import subprocess
    res = subprocess.run([sys.executable, "-c", without + "\n" + code], cwd=ROOT, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


def test_tables_of_a_captured_prune_stay(monkeypatch):
    """The positions and the mask that a captured prune reads outlive their place in the manager's cache;
    those of eager prunes do not."""
    import weakref
    import torch
    from stac_b200.stac import KVManager
    capturing = [False]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    kv = KVManager(num_layers=1, num_heads=2, head_dim=64, token_per_frame=8, buffer_size=6, chunk_size=1, recent_size=2,
                   pinned_idx=[0], device=torch.device("cuda"), dtype=torch.bfloat16)
    kv.device = torch.device("cpu")

    def tables(T, captured):
        capturing[0] = captured
        return weakref.ref(kv._base_mask(T)[0]), weakref.ref(kv._base_positions(T))
    eager, graph = tables(32, False), tables(40, True)
    assert all(t() is None for t in eager)
    again = tables(40, True)                      # a second capture finds them in the cache
    tables(48, False)
    assert all(a() is not None and a() is b() for a, b in zip(graph, again))
    assert graph[1]().tolist() == list(range(8)) + list(range(24, 40))
    assert len(kv._graph_tables) == 2


def test_snapshot_of_empty_places_reads_as_zero():
    """A snapshot of the voxel memory is zero where a row has no segment, whatever the unwritten memory
    that an empty place may point at holds."""
    import types
    import torch
    from stac_b200.stac.merger import VoxelKVMerger
    H, V, B, P, D = 2, 3, 8, 4, 64
    nan = lambda *s: torch.full(s, float("nan"))
    seg = lambda n: torch.where(torch.arange(n) < 1, 0, -1).to(torch.int32).expand(H, V, n).clone()
    seg_b, seg_p = seg(B), torch.full((H, V, P), -1, dtype=torch.int32)
    over = dict(hv=torch.zeros(1, 2, dtype=torch.int32), K=nan(1, D), V=nan(1, D), S=nan(1))
    buf = [torch.cat([torch.ones(1, *s), nan(4, *s)]) for s in ((D,), (D,), ())]
    fake = types.SimpleNamespace(
        _pull_meta=lambda: None, used_voxels=lambda: V, _meta=torch.zeros(8, dtype=torch.int32), _over=[over], _over_cur=0,
        _buf_row_seg=seg_b, _piv_row_seg=seg_p, _buf_row_cnt=torch.zeros(H, V, dtype=torch.int32),
        _piv_row_cnt=torch.zeros(H, V, dtype=torch.int32), _buf_free=torch.zeros(0, dtype=torch.int32),
        _buf_K=buf[0], _buf_V=buf[1], _buf_S=buf[2], _piv_K=nan(5, D), _piv_V=nan(5, D), _piv_W=nan(5), _piv_S=nan(5), _piv_C=nan(5))
    s = VoxelKVMerger.snapshot(fake)
    for k in ("buf_K", "buf_V", "buf_S"):
        assert (s[k][:, :, 0] == 1).all() and (s[k][:, :, 1:] == 0).all(), k
    assert all((s[k] == 0).all() for k in ("piv_K", "piv_V", "piv_W", "piv_S", "piv_C"))
