"""Parity of the tcgen05 column-sum attention against the fp32 oracle, through the C ABI.
Tolerances: output 2e-2 absolute (bf16), column sums and lse 1e-3 relative (fp32)."""

import numpy as np
import pytest
import torch

import cases
from oracle.attention import attn_colsum as oracle_attn

pytestmark = pytest.mark.gpu


def _bf16(x):
    return torch.from_numpy(x).to(torch.bfloat16)


def _run_two_segment(M, H, T_hot, T_ret, seed, T_buf=None, subsample=1.0, spread=1.0, bias_shift=0.0,
                     first_keys_scale=1.0):
    from stac_b200 import ops
    rs = np.random.RandomState(seed)
    D = 64
    T_buf = T_buf or (T_hot + 37)
    q = _bf16(rs.randn(M, H, D).astype(np.float32) * spread)
    kh_f = rs.randn(H, T_buf, D).astype(np.float32) * spread
    kh_f[:, :128] *= first_keys_scale          # the forward kernel takes its row reference from the first keys
    kh = _bf16(kh_f)
    vh = _bf16(rs.randn(H, T_buf, D).astype(np.float32))
    kr = _bf16(rs.randn(H, max(T_ret, 1), D).astype(np.float32) * spread)
    vr = _bf16(rs.randn(H, max(T_ret, 1), D).astype(np.float32))
    bias = np.log(rs.randint(1, 9, size=(H, max(T_ret, 1))).astype(np.float32))
    bias[rs.rand(H, max(T_ret, 1)) < 0.25] = -np.inf
    if bias_shift:
        bias[:, ::3] += bias_shift       # some keys far outside the usual log-count range
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    out, lse, cs = ops.attn_colsum(q.to(dev), kh.to(dev), vh.to(dev), T_hot,
                                   kr.to(dev) if T_ret else None, vr.to(dev) if T_ret else None,
                                   torch.from_numpy(bias).to(dev) if T_ret else None, T_ret,
                                   subsample_ratio=subsample, want_lse=True, status=status)
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    k_all = torch.cat([kh[:, :T_hot], kr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2)
    v_all = torch.cat([vh[:, :T_hot], vr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2)
    b_all = None
    if T_ret:
        b_all = np.concatenate([np.zeros((H, T_hot), np.float32), bias[:, :T_ret]], 1)
    o_ref, lse_ref, cs_ref = oracle_attn(q.float().numpy(), k_all, v_all, b_all, subsample_ratio=subsample)
    return (out.float().cpu().numpy(), lse.cpu().numpy(), cs.cpu().numpy()), (o_ref, lse_ref, cs_ref)


def _parts(M, H, T_hot, T_ret):
    """In how many parts each item of the call is cut on this GPU, and whether by plan a cluster joins them."""
    import ctypes
    from stac_b200 import _lib
    parts, cluster = ctypes.c_int(), ctypes.c_int()
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    assert _lib.lib().stac_attn_forward_plan(M, H, T_hot, T_ret, n_sm, 1, ctypes.byref(parts), ctypes.byref(cluster)) > 0
    return parts.value, bool(cluster.value)


def _assert_close(got, ref):
    (o, lse, cs), (o_ref, lse_ref, cs_ref) = got, ref
    assert np.isfinite(o).all() and np.isfinite(cs).all()
    assert np.abs(o - o_ref).max() <= 2e-2
    np.testing.assert_allclose(lse, lse_ref, rtol=1e-3, atol=1e-3)
    np.testing.assert_allclose(cs, cs_ref, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("M,H,T_hot,T_ret", [
    (128, 1, 128, 0),      # one tile, one warpgroup idle
    (70, 2, 200, 0),       # ragged rows and keys
    (130, 2, 236, 64),     # two query tiles, pivots with -inf padding
    (1041, 3, 1300, 200),  # frame-sized query block
    (257, 2, 0, 300),      # retrieved keys only
    (64, 1, 5, 3),         # tiny
])
def test_two_segment(M, H, T_hot, T_ret):
    got, ref = _run_two_segment(M, H, T_hot, T_ret, seed=M + T_hot)
    _assert_close(got, ref)


@pytest.mark.parametrize("T_hot,T_ret", [(50, 0), (112, 0), (113, 0), (225, 90), (336, 112), (449, 0), (460, 120), (896, 0)])
@pytest.mark.parametrize("M,H", [(130, 2), (2600, 8)])      # one CTA per item; units cut over the SMs from eight tiles on
def test_one_to_nine_key_tiles(M, H, T_hot, T_ret):
    """Fewer key tiles than score buffers, as many, one more; P V lags four tiles behind the scores."""
    _assert_close(*_run_two_segment(M, H, T_hot, T_ret, seed=T_hot + T_ret))


@pytest.mark.parametrize("T_hot,T_ret", [(336, 0), (672, 0), (600, 70), (1008, 0), (1100, 0), (1150, 90), (1400, 20)])
@pytest.mark.parametrize("M,H", [(130, 2), (2600, 8)])
def test_scores_wait_for_the_values_of_the_tile_before_them(M, H, T_hot, T_ret):
    """3, 6, 7, 9, 10, 12 and 14 key tiles, in the second shape cut over the SMs at many offsets, so that segments of every
    short length occur: scores take over the columns of probabilities only when P V has read them (same bits
    every run)."""
    got, ref = _run_two_segment(M, H, T_hot, T_ret, seed=T_hot + T_ret)
    _assert_close(got, ref)
    for _ in range(4):
        again, _ref = _run_two_segment(M, H, T_hot, T_ret, seed=T_hot + T_ret)
        assert np.array_equal(got[0], again[0]) and np.array_equal(got[1], again[1])


def test_peaked_scores():
    """Large logits exercise the running-max rescale of the online softmax."""
    got, ref = _run_two_segment(300, 2, 700, 130, seed=5, spread=3.0)
    _assert_close(got, ref)


def test_units_split_over_all_sms():
    """More (key group, head) items than SMs: the column-sum kernel cuts its units evenly over
    the SMs and items that straddle a cut are summed by two CTAs."""
    got, ref = _run_two_segment(300, 16, 3400, 140, seed=21)     # 10 key groups x 16 heads = 160 items
    _assert_close(got, ref)
    again, _ = _run_two_segment(300, 16, 3400, 140, seed=21)
    assert np.array_equal(got[2], again[2])          # shared items sum to the same bits every run


@pytest.mark.parametrize("M,H,T_hot,T_ret", [
    (130, 4, 4736, 0),      # 148 key tiles: groups of one
    (130, 4, 4737, 0),      # one tile more: groups of two, the last of a head half empty
    (70, 4, 4600, 129),     # hot and retrieved tiles in one group of two
    (130, 4, 9470, 2),      # 75 groups of two: of three
])
def test_column_sum_groups_of_one_two_and_three_tiles(M, H, T_hot, T_ret):
    _assert_close(*_run_two_segment(M, H, T_hot, T_ret, seed=M + T_hot))


def test_forward_units_split_over_all_sms():
    """More (head, query tile) items than SMs: the forward kernel runs one CTA per SM over equal
    ranges of (item, key tile) units; items on a cut are computed in two parts and joined."""
    got, ref = _run_two_segment(1200, 16, 700, 150, seed=33)
    _assert_close(got, ref)
    again, _ = _run_two_segment(1200, 16, 700, 150, seed=33)
    assert np.array_equal(got[0], again[0]) and np.array_equal(got[1], again[1])   # same bits every run


@pytest.mark.parametrize("M,H,T_hot,T_ret,spread", [(700, 2, 2500, 140, 1.0), (4164, 2, 3000, 300, 1.0),
                                                     (300, 16, 3400, 140, 2.0), (520, 3, 1777, 0, 1.0)])
def test_forward_items_cut_in_two_halves(M, H, T_hot, T_ret, spread):
    """Few heads: at most half as many (head, query tile) items as SMs and long key ranges, so every item is computed by several
    CTAs and joined: in five parts, in halves (a head-sharded stream of two heads), in three and in four."""
    assert _parts(M, H, T_hot, T_ret) == {700: (5, True), 4164: (2, True), 300: (3, False), 520: (4, True)}[M]
    got, ref = _run_two_segment(M, H, T_hot, T_ret, seed=M + H, spread=spread)
    _assert_close(got, ref)
    again, _ = _run_two_segment(M, H, T_hot, T_ret, seed=M + H, spread=spread)
    assert np.array_equal(got[0], again[0]) and np.array_equal(got[1], again[1])   # same bits every run
    assert np.array_equal(got[2], again[2])


@pytest.mark.parametrize("M,H,T_hot,T_ret", [(2600, 3, 6000, 0), (4164, 2, 5000, 300), (900, 5, 1500, 260),
                                             (1300, 1, 700, 0)])
def test_column_sums_of_items_shared_by_several_ctas(M, H, T_hot, T_ret):
    """Fewer (head, key group) items than SMs but six and more units per SM (the first two shapes):
    the column-sum units are still cut evenly over the SMs, an item is then shared by three and
    more CTAs whose partial sums meet in the workspace and are added in a fixed order (same bits
    every run).  The last two shapes stay below that and run one item per CTA."""
    got, ref = _run_two_segment(M, H, T_hot, T_ret, seed=3 * M + H)
    _assert_close(got, ref)
    for _ in range(2):
        again, _ref = _run_two_segment(M, H, T_hot, T_ret, seed=3 * M + H)
        assert np.array_equal(got[2], again[2])


def test_forward_split_with_peaked_scores():
    got, ref = _run_two_segment(1100, 16, 1000, 0, seed=34, spread=2.0)
    _assert_close(got, ref)


@pytest.mark.parametrize("M,H,T_hot", [(300, 2, 700), (1100, 16, 1000)])
def test_scores_far_above_the_first_keys(M, H, T_hot):
    """Tiny first keys give every row a reference near zero while later scores reach 2^60 and
    more above it: the kernel must notice and walk those units again with exact maxima
    (one CTA per item, and the split grid)."""
    got, ref = _run_two_segment(M, H, T_hot, 0, seed=35, spread=4.0, first_keys_scale=1e-3)
    (o, lse, cs), (o_ref, lse_ref, cs_ref) = got, ref
    assert np.isfinite(o).all() and np.isfinite(cs).all()
    assert np.abs(o - o_ref).max() <= 2e-2 * max(1.0, float(np.abs(o_ref).max()))
    np.testing.assert_allclose(lse, lse_ref, rtol=1e-3, atol=1e-3)
    np.testing.assert_allclose(cs, cs_ref, rtol=1e-3, atol=1e-6)


def test_one_key_far_above_the_first_keys():
    """A single key 2^144 above the row reference, at every place of a chunk of 32: whichever pipe its exponential runs on,
    the CTA walks its units again with exact maxima (one call per place)."""
    from stac_b200 import ops
    rs = np.random.RandomState(8)
    M, T, dev = 40, 300, torch.device("cuda:0")
    u = rs.randn(64).astype(np.float32)
    u /= np.linalg.norm(u)
    q = _bf16(8 * u + 0.1 * rs.randn(M, 1, 64).astype(np.float32))
    v = _bf16(rs.randn(1, T, 64).astype(np.float32))
    for place in range(224, 224 + 32):
        k = rs.randn(1, T, 64).astype(np.float32)
        k[0, place] = 100 * u
        k = _bf16(k)
        got = ops.attn_colsum(q.to(dev), k.to(dev), v.to(dev), T, want_lse=True)
        ref = oracle_attn(q.float().numpy(), k.float().numpy().transpose(1, 0, 2), v.float().numpy().transpose(1, 0, 2), None)
        _assert_close([x.float().cpu().numpy() for x in got], ref)


@pytest.mark.parametrize("M,H,T_hot,T_ret", [
    (130, 3, 300, 0),        # one CTA per item, a segment of three tiles
    (130, 2, 449, 130),      # a tile of one key, masked pivots
    (2600, 16, 800, 150),    # items cut over the SMs: parts of all lengths, several segments per CTA
    (1100, 2, 2000, 100),    # items in five parts
    (4164, 2, 1200, 100),    # items in halves
])
@pytest.mark.parametrize("first,last", [(0.4, 0.6), (0.97, 1.0), (0.2, 1.0)])       # where the keys are that are far from the others
def test_some_segments_are_walked_twice(M, H, T_hot, T_ret, first, last):
    """Keys of the first head, and of the last one, that are 20 times as long as the others, whichever part of an item they lie in: rows of
    their CTAs outgrow their references.  Another CTA's rows have the bits that they have without such keys, a second call those of the first."""
    from stac_b200 import ops
    rs = np.random.RandomState(M + T_hot)
    q, k, v, kr, vr = (rs.randn(*s).astype(np.float32) for s in ((M, H, 64),) + ((H, T_hot, 64),) * 2 + ((H, T_ret + 1, 64),) * 2)
    a, b = int(T_hot * first), max(int(T_hot * first) + 1, int(T_hot * last))
    plain = _bf16(k)
    k[[0, H - 1], a:b] *= 20
    q, k, v, kr, vr = (_bf16(2 * q), _bf16(k), _bf16(v), _bf16(kr), _bf16(vr))
    bias = np.log(rs.randint(1, 9, size=(H, T_ret + 1)).astype(np.float32))
    bias[:, :T_ret // 2] = -np.inf
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    ret = (kr.to(dev), vr.to(dev), torch.from_numpy(bias).to(dev), T_ret) if T_ret else (None, None, None, 0)
    got, again, unflagged = (ops.attn_colsum(q.to(dev), x.to(dev), v.to(dev), T_hot, *ret, want_lse=True, status=status)
                             for x in (k, k, plain))
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    assert all(torch.equal(x, y) for x, y in zip(got, again))
    if H == 3:       # no CTA has rows of two heads
        assert torch.equal(got[1][1:-1], unflagged[1][1:-1]) and torch.equal(got[0][:, 1:-1], unflagged[0][:, 1:-1])
    o_ref, lse_ref, cs_ref = oracle_attn(q.float().numpy(), torch.cat([k, kr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2),
                                         torch.cat([v, vr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2),
                                         np.concatenate([np.zeros((H, T_hot), np.float32), bias[:, :T_ret]], 1))
    o, lse, cs = (x.float().cpu().numpy() for x in got)
    assert np.abs(o - o_ref).max() <= 2e-2 * max(1.0, float(np.abs(o_ref).max()))
    np.testing.assert_allclose(lse, lse_ref, rtol=1e-3, atol=1e-3)
    np.testing.assert_allclose(cs, cs_ref, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("M,H,T_hot,T_ret", [
    (64, 1, 12 * 112, 0),        # one item, four parts of three tiles, joined by a cluster
    (1, 1, 11 * 112 + 1, 90),    # a tile of one key among the parts' ends
    (300, 2, 2500, 260),         # six items
    (130, 3, 150, 6000),         # mostly retrieved keys, a cluster of eight
    (128, 1, 40000, 0),          # more parts than a cluster has CTAs: through the workspace
    (257, 6, 9000, 100),         # clusters of six
    (700, 8, 2000, 0),           # more items than clusters of the best size: through the workspace, 48 items in three parts
    (128, 2, 40000, 0),          # two items of twenty parts through the workspace
    (4164, 2, 3000, 300),        # 66 items in halves, a stream of two heads
])
@pytest.mark.parametrize("kind", ["plain", "far", "masked"])
def test_items_in_many_parts(M, H, T_hot, T_ret, kind):
    """Few items: each is cut in equal parts, which a cluster or whoever comes last adds up.  far: keys 20 times as long as the others in the middle,
    so that the CTAs of some parts walk twice; masked: nearly all retrieved keys are, whole parts among them.  A second call has the same bits."""
    from stac_b200 import ops
    rs = np.random.RandomState(M + T_hot)
    n_ret = max(T_ret, 1)
    q, k, v, kr, vr = (rs.randn(*s).astype(np.float32) for s in ((M, H, 64), (H, T_hot, 64), (H, T_hot, 64), (H, n_ret, 64), (H, n_ret, 64)))
    if kind == "far":
        k[0, T_hot // 2:T_hot // 2 + 40] *= 20
        q *= 2
    bias = np.log(rs.randint(1, 9, size=(H, n_ret)).astype(np.float32))
    if kind == "masked":
        bias[:, n_ret // 50 + 1:] = -np.inf
    q, k, v, kr, vr = (_bf16(x) for x in (q, k, v, kr, vr))
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    ret = (kr.to(dev), vr.to(dev), torch.from_numpy(bias).to(dev), T_ret) if T_ret else (None, None, None, 0)
    assert _parts(M, H, T_hot, T_ret) == {(64, 1): (4, True), (1, 1): (5, True), (300, 2): (7, True), (130, 3): (8, True), (128, 1): (20, False),
                                          (257, 6): (6, True), (700, 8): (3, False), (128, 2): (20, False), (4164, 2): (2, True)}[M, H]
    got, again = (ops.attn_colsum(q.to(dev), k.to(dev), v.to(dev), T_hot, *ret, want_lse=True, status=status) for _ in range(2))
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    assert all(torch.equal(x, y) for x, y in zip(got, again))
    o_ref, lse_ref, cs_ref = oracle_attn(q.float().numpy(), torch.cat([k, kr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2),
                                         torch.cat([v, vr[:, :T_ret]], 1).float().numpy().transpose(1, 0, 2),
                                         np.concatenate([np.zeros((H, T_hot), np.float32), bias[:, :T_ret]], 1))
    o, lse, cs = (x.float().cpu().numpy() for x in got)
    assert np.abs(o - o_ref).max() <= 2e-2 * max(1.0, float(np.abs(o_ref).max()))
    np.testing.assert_allclose(lse, lse_ref, rtol=1e-3, atol=1e-3)
    np.testing.assert_allclose(cs, cs_ref, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("what", ["key", "bias"])
def test_nan_at_every_place(what):
    """A NaN key, or a NaN bias of a pivot, at every place of a chunk of 32: every output row of its head is NaN, whichever pipe its
    exponential runs on, and the other head's are not."""
    from stac_b200 import ops
    M, T, dev = 40, 336, torch.device("cuda:0")      # whole tiles of 112 keys
    g = torch.Generator().manual_seed(3)
    q, k, v, kr, vr = (torch.randn(*s, generator=g).to(torch.bfloat16).to(dev) for s in ((M, 2, 64),) + ((2, T, 64),) * 4)
    for place in range(128, 128 + 32):
        k2, br = k.clone(), torch.zeros(2, T, device=dev)
        if what == "key":
            k2[0, place] = float("nan")
        else:
            br[0, place] = float("nan")
        out, lse, _ = ops.attn_colsum(q, k2, v, T, kr, vr, br, T, want_lse=True)
        assert out[:, 0].isnan().all() and lse[0].isnan().all(), place
        assert out[:, 1].isfinite().all() and lse[1].isfinite().all(), place


@pytest.mark.parametrize("shift", [-40.0, 30.0])
def test_large_bias(shift):
    got, ref = _run_two_segment(200, 2, 300, 260, seed=13, bias_shift=shift)
    _assert_close(got, ref)


@pytest.mark.parametrize("ratio", [0.25, 0.5])
def test_subsampled_colsum(ratio):
    got, ref = _run_two_segment(1041, 2, 900, 0, seed=9, subsample=ratio)
    _assert_close(got, ref)


@pytest.mark.parametrize("name", list(cases.ATTENTION))
def test_reference_layout_entry(name, golden_dir):
    """flash_attn_bias_colsum with the reference's [B,T,H,D] tensors against the committed
    torch-generated fixture."""
    import os
    from stac_b200 import ops
    g = np.load(os.path.join(golden_dir, "attention.npz"))
    q, k, v, bias = cases.attention_inputs(name)
    dev = torch.device("cuda:0")
    tq, tk, tv = (_bf16(x)[None].to(dev) for x in (q, k, v))
    tb = None if bias is None else torch.from_numpy(bias)[None, :, None, :].to(dev)
    out, lse, cs = ops.flash_attn_bias_colsum(tq, tk, tv, bias=tb, return_colsum=True)
    torch.cuda.synchronize()
    assert np.abs(out[0].float().cpu().numpy() - g[f"{name}_out"]).max() <= 2e-2
    np.testing.assert_allclose(lse[0].cpu().numpy(), g[f"{name}_lse"], rtol=1e-3, atol=1e-3)
    np.testing.assert_allclose(cs[0].cpu().numpy(), g[f"{name}_colsum"], rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("name", list(cases.ATTENTION_REF))
def test_against_the_reference_kernels(name, golden_dir):
    """The CUDA path against what the reference's own Triton kernels returned on a B200 for the
    same seeded inputs (attention_ref.npz, made by tests/golden/make_attention_ref.py): O within
    2e-2, lse and column sums within 1e-3 relative.  Where the Triton entry point sub-samples
    rows differently from the reference's CUDA backend (M not a multiple of 128), the column sums
    are held to the oracle, which the CPU tests hold to the same fixture with that rule."""
    import os
    from stac_b200 import ops
    g = np.load(os.path.join(golden_dir, "attention_ref.npz"))
    c = cases.ATTENTION_REF[name]
    q, k, v, bias = cases.attention_inputs(name)
    dev = torch.device("cuda:0")
    tq, tk, tv = (_bf16(x)[None].to(dev) for x in (q, k, v))
    tb = None if bias is None else torch.from_numpy(bias)[None, :, None, :].to(dev)
    out, lse, cs = ops.flash_attn_bias_colsum(tq, tk, tv, bias=tb, return_colsum=True, subsample_ratio=c["ratio"])
    torch.cuda.synchronize()
    o_ref = (g[f"{name}_out_bf16"].view(np.uint16).astype(np.uint32) << 16).view(np.float32)
    assert np.abs(out[0].float().cpu().numpy() - o_ref).max() <= 2e-2
    np.testing.assert_allclose(lse[0].cpu().numpy(), g[f"{name}_lse"], rtol=1e-3, atol=1e-3)
    if c["same_rule"]:
        cs_ref = g[f"{name}_colsum"]
    else:
        _, _, cs_ref = oracle_attn(q, k, v, bias, subsample_ratio=c["ratio"])
    np.testing.assert_allclose(cs[0].cpu().numpy(), cs_ref, rtol=1e-3, atol=1e-6)
    # the two-segment entry (hot keys | biased pivots) on the same data
    n_b = c["n_bias"]
    if n_b and n_b < c["N"]:
        T_hot = c["N"] - n_b
        kh, vh = tk[0].transpose(0, 1).contiguous(), tv[0].transpose(0, 1).contiguous()      # [H,N,D]
        o2, lse2, cs2 = ops.attn_colsum(tq[0], kh, vh, T_hot, kh[:, T_hot:].contiguous(), vh[:, T_hot:].contiguous(),
                                        torch.from_numpy(bias[:, T_hot:]).contiguous().to(dev), n_b,
                                        subsample_ratio=c["ratio"], want_lse=True)
        torch.cuda.synchronize()
        assert np.abs(o2.float().cpu().numpy() - o_ref).max() <= 2e-2
        np.testing.assert_allclose(lse2.cpu().numpy(), g[f"{name}_lse"], rtol=1e-3, atol=1e-3)
        np.testing.assert_allclose(cs2.cpu().numpy(), cs_ref, rtol=1e-3, atol=1e-6)


def test_leading_masked_tile_then_faint_keys():
    """The first key tile of the biased segment is all padding (-inf) and the live keys behind it
    carry a large negative bias: the row reference must come from live keys, not from the masked
    tile, or every probability underflows."""
    from stac_b200 import ops
    rs = np.random.RandomState(17)
    M, H, D, N = 150, 2, 64, 400
    q = _bf16(rs.randn(M, H, D).astype(np.float32))
    k = _bf16(rs.randn(H, N, D).astype(np.float32))
    v = _bf16(rs.randn(H, N, D).astype(np.float32))
    bias = np.full((H, N), -200.0, np.float32)
    bias[:, :112] = -np.inf
    bias[:, 300:] = -np.inf
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    out, lse, cs = ops.attn_colsum(q.to(dev), None, None, 0, k.to(dev), v.to(dev), torch.from_numpy(bias).to(dev), N,
                                   want_lse=True, status=status)
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    o_ref, lse_ref, cs_ref = oracle_attn(q.float().numpy(), k.float().numpy().transpose(1, 0, 2),
                                         v.float().numpy().transpose(1, 0, 2), bias)
    _assert_close((out.float().cpu().numpy(), lse.cpu().numpy(), cs.cpu().numpy()), (o_ref, lse_ref, cs_ref))


@pytest.mark.parametrize("M,H,N", [(70, 2, 1), (130, 2, 112), (130, 3, 449), (257, 2, 1000), (2600, 8, 900), (1100, 2, 2000)])
@pytest.mark.parametrize("kind", ["counts", "mask", "lowest", "faint", "huge", "scale"])
def test_a_bias_on_every_key(M, H, N, kind):
    """Log counts with masked keys and whole masked tiles (first, middle, last of a head), a type's lowest value and a finite one
    within its range as the mask, biases that swallow the scores, a scale that is not a power of two.  One CTA per item,
    items cut over the SMs, items in halves."""
    from stac_b200 import ops
    rs = np.random.RandomState(M + N)
    q, k, v = (_bf16(rs.randn(*s).astype(np.float32)) for s in ((M, H, 64), (N, H, 64), (N, H, 64)))
    bias = np.log(rs.randint(1, 9, size=(H, N)).astype(np.float32))
    scale = 0.1 if kind == "scale" else 0.125
    if kind == "huge":
        bias -= np.float32(3e37)
    elif kind != "counts" and N > 1:
        masked = rs.rand(H, N) < 0.25
        for h, tile in ((0, 0), (1, 3), (H - 1, (N - 1) // 112)):
            masked[h, 112 * tile:112 * (tile + 1)] = N > 112
        bias[masked] = {"lowest": np.finfo(np.float32).min, "faint": np.float32(-3e37)}.get(kind, -np.inf)
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    got = ops.attn_colsum(q.to(dev), None, None, 0, k.to(dev), v.to(dev), torch.from_numpy(bias).to(dev), N, layout="thd",
                          scale=scale, want_lse=True, status=status)
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    o, lse, cs = oracle_attn(q.float().numpy(), k.float().numpy(), v.float().numpy(), bias, scale=scale)
    if kind == "huge":
        cs = np.zeros_like(cs)       # rows whose log-sum-exp is beyond 1e29 add nothing to the column sums
    _assert_close([x.float().cpu().numpy() for x in got], (o, lse, cs))


@pytest.mark.parametrize("shift", [-40.0, 30.0, 300.0])
@pytest.mark.parametrize("scale", [0.125, 0.1])
def test_a_bias_far_from_zero_is_added_behind_the_scale(shift, scale):
    """One rounding of the exponents at the bias's size.  Column sums: half an ulp of the biased exponent and half an ulp of the
    row's log-sum-exp, both in log2 units, beside a quarter of the cubic's mean error (8.24e-6).  Log-sum-exps: four
    such roundings (bias, exponent, sum with the reference, change of base) beside 1.4e-5 for the cubic in an eighth of 300 keys."""
    from stac_b200 import ops
    M, N, H = 500, 300, 4
    rs = np.random.RandomState(21)
    q, k, v = (_bf16(rs.randn(*s).astype(np.float32)) for s in ((M, H, 64), (N, H, 64), (N, H, 64)))
    bias = np.log(rs.randint(1, 9, size=(H, N))).astype(np.float32) + np.float32(shift)
    dev = torch.device("cuda:0")
    _, lse, cs = ops.attn_colsum(q.to(dev), None, None, 0, k.to(dev), v.to(dev), torch.from_numpy(bias).to(dev), N, layout="thd",
                                 scale=scale, want_lse=True)
    s = torch.einsum("mhd,nhd->hmn", q.double(), k.double()) * scale + torch.from_numpy(bias).double()[:, None]
    lse_ref = s.logsumexp(-1)
    cs_ref = (s - lse_ref[..., None]).exp().sum(1)
    rounding = float(np.spacing(np.float32(abs(shift) * 1.4427))) * 0.6931
    assert ((cs.cpu().double() - cs_ref).norm() / cs_ref.norm()).item() <= 2.1e-6 + rounding
    assert (lse.cpu().double() - lse_ref).abs().max().item() <= 1.4e-5 + 2 * rounding


def test_calls_replay_from_a_cuda_graph():
    """The entry point neither allocates nor synchronises, so calls can be captured into a CUDA
    graph (the programmatic-serialization edges between its kernels included); a replay gives the
    bits of the eager call."""
    from stac_b200 import ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(12)
    M, H, T_hot, T_ret, D = 700, 4, 2000, 150, 64
    q = (torch.randn(M, H, D, generator=g) / 2).to(torch.bfloat16).to(dev)
    kh = (torch.randn(H, T_hot, D, generator=g) / 2).to(torch.bfloat16).to(dev)
    vh = torch.randn(H, T_hot, D, generator=g).to(torch.bfloat16).to(dev)
    kr = (torch.randn(H, T_ret, D, generator=g) / 2).to(torch.bfloat16).to(dev)
    vr = torch.randn(H, T_ret, D, generator=g).to(torch.bfloat16).to(dev)
    bias = torch.log(torch.randint(1, 9, (H, T_ret), generator=g).float()).to(dev)
    status = ops.DeviceStatus(dev)

    def call():
        return ops.attn_colsum(q, kh, vh, T_hot, kr, vr, bias, T_ret, want_lse=True, status=status)
    side = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(side):
        eager = [t.clone() for t in call()]          # also sizes the workspace of this stream
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            first = call()
            second = call()
        for t in first + second:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
    status.raise_if_set("graph replay")
    for a, b, c in zip(eager, first, second):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("warm", [True, False])     # eager calls made before on the stream of the capture, or not
@pytest.mark.parametrize("M,H,T_hot", [(700, 4, 2000), (2600, 16, 700)])   # parts joined at cuts: column sums; forward
def test_replay_after_the_eager_workspace_was_replaced(M, H, T_hot, warm):
    """A larger eager call on the stream of the capture replaces the workspace kept for that stream, other
    tensors take its memory: a replay still gives the eager bits, and writes to none of them."""
    from stac_b200 import ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(21)

    def inputs(M, H, T):
        return [torch.randn(*s, generator=g).to(torch.bfloat16).to(dev) for s in ((M, H, 64), (H, T, 64), (H, T, 64))]
    q, k, v = inputs(M, H, T_hot)
    big = inputs(2 * M, 2 * H, T_hot)
    status = ops.DeviceStatus(dev)
    eager = ops.attn_colsum(q, k, v, T_hot, want_lse=True, status=status)
    torch.cuda.synchronize()
    side = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(side):
        if warm:
            ops.attn_colsum(q, k, v, T_hot, want_lse=True, status=status)
            torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            captured = ops.attn_colsum(q, k, v, T_hot, want_lse=True, status=status)
        size = ops._attn_workspace(dev, M, H).numel()
        ops.attn_colsum(big[0], big[1], big[2], T_hot, status=status)
        others = [torch.full((size,), 3.0, device=dev) for _ in range(4)]
        for _ in range(2):
            for t in captured:
                t.zero_()
            graph.replay()
            torch.cuda.synchronize()
            for a, b in zip(eager, captured):
                assert torch.equal(a, b)
        assert all(bool((t == 3.0).all()) for t in others)
    status.raise_if_set("graph replay")
    torch.cuda.synchronize()


def test_bounded_wait_reports_and_returns():
    """A wait on a barrier nothing completes runs out, sets the status word and the kernel
    returns; the context stays usable."""
    from stac_b200 import _lib, ops
    dev = torch.device("cuda:0")
    status = ops.DeviceStatus(dev)
    rc = _lib.lib().stac_selftest_bounded_wait(2000, _lib.ptr(status.word), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    assert status.read() == 6
    status.clear()
    assert float(torch.ones(4, device=dev).sum().item()) == 4.0


@pytest.mark.parametrize("M,Lk,pivots", [(4164, 17700, 2082), (1041, 33312, 0)])
def test_full_size_against_torch_fp32(M, Lk, pivots):
    """The stream shape (one 4-frame chunk against the full hot cache plus retrieved pivots) and the
    longest microbenchmark shape are too large for the numpy oracle: same checks against a plain
    torch fp32 restatement on the device, four heads at a time; and the same bits on a second run."""
    from stac_b200 import ops
    dev = torch.device("cuda:0")
    g = torch.Generator(device="cpu").manual_seed(77)
    H, D = 16, 64
    q = (torch.randn(M, H, D, generator=g) / 2).to(torch.bfloat16).to(dev)
    k = (torch.randn(H, Lk, D, generator=g) / 2).to(torch.bfloat16).to(dev)
    v = (torch.randn(H, Lk, D, generator=g) / 8).to(torch.bfloat16).to(dev)
    T_hot = Lk - pivots
    bias = kr = vr = None
    if pivots:
        bias = torch.log(torch.randint(1, 9, (H, pivots), generator=g).float())
        bias[torch.rand(H, pivots, generator=g) < 0.25] = float("-inf")
        bias = bias.to(dev)
        kr, vr = k[:, T_hot:].contiguous(), v[:, T_hot:].contiguous()
    status = ops.DeviceStatus(dev)
    runs = [ops.attn_colsum(q, k, v, T_hot, kr, vr, bias, pivots, want_lse=True, status=status) for _ in range(2)]
    torch.cuda.synchronize()
    status.raise_if_set("attention")
    out, lse, cs = runs[0]
    assert all(torch.equal(a, b) for a, b in zip(runs[0], runs[1]))
    for h0 in range(0, H, 4):
        s = torch.einsum("mhd,hnd->hmn", q[:, h0:h0 + 4].float(), k[h0:h0 + 4].float()) * D ** -0.5
        if pivots:
            s[:, :, T_hot:] += bias[h0:h0 + 4, None, :]
        p = torch.softmax(s, -1)
        o_ref = torch.einsum("hmn,hnd->mhd", p, v[h0:h0 + 4].float())
        assert float((out[:, h0:h0 + 4].float() - o_ref).abs().max()) <= 2e-2
        torch.testing.assert_close(cs[h0:h0 + 4], p.sum(1), rtol=1e-3, atol=1e-6)
        torch.testing.assert_close(lse[h0:h0 + 4], torch.logsumexp(s, -1), rtol=1e-3, atol=1e-3)
        del s, p


def test_kept_workspace_between_calls_of_all_kinds():
    """The kept workspace is zeroed once: every call, of any size and on either walk of the forward kernel (a call
    whose units are walked again included, with and without column sums), has to leave its control
    words zero, and gives the bits of the entry that clears a workspace full of rubbish."""
    from stac_b200 import _lib, ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(3)
    p = _lib.ptr
    #        M, H, T_hot, scale of the keys behind the first tile, column sums
    calls = [(300, 2, 700, 1.0, True), (1100, 16, 1000, 20.0, True), (300, 16, 3400, 1.0, True), (64, 1, 5, 1.0, False),
             (300, 2, 700, 20.0, False), (700, 2, 2500, 20.0, True), (2600, 3, 6000, 1.0, True), (300, 2, 700, 1.0, True)]
    for M, H, T, far, want in calls:
        q = torch.randn(M, H, 64, generator=g).to(torch.bfloat16).to(dev)
        k = torch.randn(H, T, 64, generator=g)
        k[:, 128:] *= far
        k = k.to(torch.bfloat16).to(dev)
        v = torch.randn(H, T, 64, generator=g).to(torch.bfloat16).to(dev)
        out, lse, cs = ops.attn_colsum(q, k, v, T, want_lse=True, want_colsum=want)
        ws = ops._attn_workspace(dev, M, H)
        assert int(ws[:ops.ATTN_CTL_WORDS].view(torch.int32).abs().sum().item()) == 0
        out2, lse2 = torch.empty_like(out), torch.empty_like(lse)
        cs2 = torch.empty_like(cs) if want else None
        rubbish = torch.full((_lib.lib().stac_attn_workspace_bytes(M, H) // 4,), 3.0, device=dev)
        rc = _lib.lib().stac_attn_colsum(
            p(q), q.stride(0), p(k), p(v), k.stride(1), k.stride(0), T, None, None, 64, 64, 0, None, 0, p(out2),
            out2.stride(0), p(lse2), p(cs2), T, M, H, 64, 0.125, 1.0, p(rubbish), rubbish.numel() * 4, None,
            _lib.stream_ptr())
        assert rc == 0
        assert torch.equal(out, out2) and torch.equal(lse, lse2)
        assert not want or torch.equal(cs, cs2)


@pytest.mark.parametrize("M", [1, 15, 16, 17, 48, 49, 63, 64, 65, 80, 112, 127, 128 + 1, 128 + 64, 128 + 65, 1041])
@pytest.mark.parametrize("H,T_hot,T_ret", [(2, 300, 90), (16, 3400, 140)])     # one CTA per item; units cut over the SMs
def test_ragged_last_query_tile(M, H, T_hot, T_ret):
    """Column sums score only the halves of the last query tile that hold rows, and of the last half only
    the 16-row pieces up to the last row; a bias out of the usual range takes the other exponent path."""
    for shift in (0.0, -40.0):
        got, ref = _run_two_segment(M, H, T_hot, T_ret, seed=M, bias_shift=shift)
        _assert_close(got, ref)


@pytest.mark.parametrize("M,H,T_hot,T_ret,old_T,ratio", [
    (130, 2, 300, 90, 170, 1.0),          # one CTA per item: updated by the kernel
    (1041, 16, 3400, 140, 2359, 1.0),     # one to two items per SM, nearly all shared by two CTAs: by the thread that adds second
    (2600, 3, 6000, 0, 0, 1.0),           # by three and more: by the CTA that joins them
    (900, 5, 1500, 260, 1500, 0.25),      # rows left out; no new key
    (2600, 3, 5900, 200, 4000, 1.0),      # hot and retrieved tiles in one group of items shared by three CTAs
    (300, 16, 7300, 200, 5000, 1.0),      # two and more items per SM, some shared by two CTAs
])
def test_scores_updated_by_the_column_sum_kernel(M, H, T_hot, T_ret, old_T, ratio):
    """The running scores and counts get the bits that the update behind the call gives; the other outputs, the keys
    behind the live ones and the retrieved keys are left alone."""
    from stac_b200 import _lib, ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(M + H)
    q, k, v = (torch.randn(*shape, generator=g).to(torch.bfloat16).to(dev) for shape in
               ((M, H, 64), (H, T_hot + 37, 64), (H, T_hot + 37, 64)))
    kr, vr = (torch.randn(H, max(T_ret, 1), 64, generator=g).to(torch.bfloat16).to(dev) for _ in range(2))
    br = torch.log(torch.randint(1, 9, (H, max(T_ret, 1)), generator=g).float()).to(dev)
    ret = (kr, vr, br, T_ret) if T_ret else (None, None, None, 0)
    width = T_hot + 50
    scores, counts = (torch.rand(H, width, generator=g).to(dev) for _ in range(2))
    want_s, want_c = scores.clone(), counts.clone()
    out, lse, cs = ops.attn_colsum(q, k, v, T_hot, *ret, want_lse=True, subsample_ratio=ratio)
    rc = _lib.lib().stac_scores_update(_lib.ptr(cs), cs.stride(0), _lib.ptr(want_s), _lib.ptr(want_c), width, H, T_hot, old_T,
                                       M, 0.9, _lib.stream_ptr())
    assert rc == 0
    for _ in range(2):        # the second call finds the workspace as the first one leaves it
        s2, c2 = scores.clone(), counts.clone()
        got = ops.attn_colsum(q, k, v, T_hot, *ret, want_lse=True, subsample_ratio=ratio, score_update=(s2, c2, width, old_T, M, 0.9))
        assert all(torch.equal(a, b) for a, b in zip(got, (out, lse, cs)))
        assert torch.equal(s2, want_s) and torch.equal(c2, want_c)
