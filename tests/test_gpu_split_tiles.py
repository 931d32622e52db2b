"""Packed decode pipeline: even and odd tiles of a row on warp groups of their own, k-steps and copies cut at the tile's longest
row.  Rows of one to five tiles per CTA in every phase of the rings, tiles of short rows only, tiles whose K or V rows are all
empty, single long rows among short ones, scores that raise the reference maximum in one group only."""
import ctypes

import pytest
import torch

from dynakv_b200 import _lib, synthetic
from dynakv_b200.kernels import _common
from oracle import dynakv_oracle as O

pytestmark = pytest.mark.gpu


def _row_errors(out, ref):
    """Relative 2-norm of the error of each (row, head)."""
    return (out.float().cpu() - ref).norm(dim=-1) / ref.norm(dim=-1).clamp_min(1e-30)


def _row_limit(dtype, spread=1.0):
    """A result is off by the roundings of the result, of the weights and of the rotated keys and queries, each by at most half a
    unit u in the last place and independent over tokens and dimensions: u (1 + 1 + 2 s) for scores that spread by s (queries of
    unit variance: about 1).  Losing 32 tokens of any row here
    changes a head's result by 1.8 times as much or more."""
    return (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -11) * (2 + 2 * spread)


def _decode(c, lens_k, lens_v, n_sm, theta=5e5, knorm=None, spread=1.0):
    """dkv_two_stage_decode on `n_sm` SMs: the fewer, the more tiles a CTA walks."""
    gen = torch.Generator().manual_seed(3)
    k, v = (synthetic.ragged_side(x, gen, c.q.dtype) for x in (lens_k, lens_v))
    args = [c.q, k.flat, c.k_up, v.flat, c.v_up, k.lens, k.offs, v.lens, v.offs]
    ref = O.compact_attention(*args[:5], *args[5:], theta, seq_lens=c.seq_lens, k_norm_weight=knorm)
    d = [t.cuda() for t in args]
    out = torch.zeros(c.q.shape, dtype=c.q.dtype, device="cuda")
    a, keep = _common.build_attn_args(d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], d[8], theta, out=out, len_multiple=8, need_workspace=True,
                                      seq_lens=torch.tensor(c.seq_lens, dtype=torch.int32, device="cuda"),
                                      k_norm_weight=None if knorm is None else knorm.cuda())
    a.n_sm = n_sm
    need = int(_lib.load().dkv_split_workspace_bytes(ctypes.byref(a)))
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    _lib.check(_lib.load().dkv_two_stage_decode(ctypes.byref(a)), "dkv_two_stage_decode")
    torch.cuda.synchronize()
    del keep
    assert float(_row_errors(out, torch.nan_to_num(ref)).max()) <= _row_limit(c.q.dtype, spread)
    assert _common.read_status(torch.device("cuda")) == 0


def _lengths(kind, rows, S, gen):
    lens = torch.randint(1, 17, (rows, S), generator=gen, dtype=torch.int32) * 8
    if kind == "short":
        lens = lens.clamp(max=16)
    elif kind == "one long":
        lens = lens.clamp(max=24)
        lens[:, S // 2] = 128
    elif kind == "empty tiles":
        lens[:, 128:256] = 0
        lens[:, 300:] = 0
    return lens


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("kind", ["any", "short", "one long", "empty tiles"])
@pytest.mark.parametrize("seq,n_sm", [([640], 2), ([1, 128, 129, 257, 513], 2), ([385, 1, 640, 256, 3], 6),
                                      ([300, 257, 129, 640, 200, 385, 513, 256, 300], 2)], ids=str)
def test_tiles_of_both_groups(seq, n_sm, kind, dtype):
    gen = torch.Generator().manual_seed(len(seq) + n_sm)
    c = synthetic.make_layer_case(7, seq, "uniform", 5e5, dtype, "cpu", n_q_heads=8, n_kv_heads=2)
    lens_k, lens_v = (_lengths(kind, 2 * len(seq), max(seq), gen) for _ in range(2))
    _decode(c, lens_k, lens_v, n_sm, knorm=1.0 + 0.1 * torch.randn(128, generator=gen) if kind == "any" else None)


@pytest.mark.parametrize("tile", [0, 1, 3, 4])
def test_reference_maximum_raised_in_one_group(tile):
    gen = torch.Generator().manual_seed(11)
    c = synthetic.make_layer_case(9, [640], "uniform", 5e5, torch.bfloat16, "cpu", n_q_heads=8, n_kv_heads=2)
    c.q[:, :] *= 4
    lens = torch.full((2, 640), 8, dtype=torch.int32)
    lens[:, 128 * tile:128 * tile + 128] = 128
    _decode(c, lens, lens.flip(1).contiguous(), 2, spread=4.0)


@pytest.mark.parametrize("switch", [500, 64])
@pytest.mark.parametrize("seq", [[1024, 1, 499, 500], [1025, 1, 499, 500], [0, 700, 3], [130] * 20 + [900]], ids=["1024", "1025", "empty", "21 rows"])
def test_routes_of_a_routed_call(seq, switch):
    """One route for all rows, both sides of its lines, and the three kernels between; bounds left in the arguments are ignored."""
    c = synthetic.make_layer_case(21, seq, "beta:2,5", 5e5, torch.bfloat16, "cpu", n_q_heads=16, n_kv_heads=4)
    fk, fv, lk, lv, ok, ov = c.views()
    ref = torch.nan_to_num(O.compact_attention(c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov, c.theta, seq_lens=seq))
    d = [t.cuda() for t in (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)]
    out = torch.full(c.q.shape, 7.0, dtype=c.q.dtype, device="cuda")
    a, keep = _common.build_attn_args(*d, c.theta, out=out, len_multiple=8, need_workspace=True, route_min_tokens=5, route_max_tokens=9,
                                      seq_lens=torch.tensor(seq, dtype=torch.int32, device="cuda"))
    _lib.check(_lib.load().dkv_routed_decode(ctypes.byref(a), switch), "dkv_routed_decode")
    assert _lib.load().dkv_routed_launches(ctypes.byref(a), switch) == (1 if max(seq) <= {500: 1024, 64: 256}[switch] and len(seq) < 9 else 2 if len(seq) > 9 and switch == 500 else 3)
    assert float(_row_errors(out, ref).max()) <= _row_limit(torch.bfloat16)
    assert _common.read_status(torch.device("cuda")) == (4 if 0 in seq else 0)      # an empty row is reported
    del keep


def _run(c, entry, n_sm, switch=None, repeats=30, **more):
    """An entry on `n_sm` SMs, its result and the status; repeated runs have to agree bit for bit."""
    fk, fv, lk, lv, ok, ov = c.views()
    ref = torch.nan_to_num(O.compact_attention(c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov, c.theta, seq_lens=c.seq_lens))
    d = [t.cuda() for t in (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)]
    out = torch.full(c.q.shape, 7.0, dtype=c.q.dtype, device="cuda")
    a, keep = _common.build_attn_args(*d, c.theta, out=out, len_multiple=8, need_workspace=True,
                                      seq_lens=torch.tensor(c.seq_lens, dtype=torch.int32, device="cuda"), **more)
    a.n_sm = n_sm
    ws = torch.empty(int(_lib.load().dkv_split_workspace_bytes(ctypes.byref(a))), dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    first = None
    for _ in range(repeats):
        out.fill_(7.0)
        _lib.check(entry(ctypes.byref(a)) if switch is None else entry(ctypes.byref(a), switch), "attention")
        first = out.clone() if first is None else first
        assert torch.equal(out, first)
    del keep
    return a, first, ref, _common.read_status(torch.device("cuda"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("n_sm", [2, 4, 6])
@pytest.mark.parametrize("seq", [[100, 0, 300], [0, 0, 700], [129, 0, 0, 1, 0, 257], [640, 0, 128, 0, 0, 384, 0], [256, 0, 90, 0, 1000, 0, 0, 5] * 2], ids=str)
def test_rows_without_tiles_between_others(seq, n_sm, dtype):
    """A CTA that goes from one row over rows without tiles to another one, or to its end."""
    c = synthetic.make_layer_case(13, seq, "beta:2,5", 5e5, dtype, "cpu", n_q_heads=8, n_kv_heads=2)
    _, out, ref, status = _run(c, _lib.load().dkv_two_stage_decode, n_sm)
    empty = torch.tensor(seq) == 0
    assert float(out[empty.cuda()].abs().max()) == 0 and status == 4      # an empty row is reported
    assert float(_row_errors(out, ref)[~empty].max()) <= _row_limit(dtype)


@pytest.mark.parametrize("n_sm", [8, 10, 14])
@pytest.mark.parametrize("seq", [[1300, 40, 500, 63, 7, 1200, 128, 1], [1, 64, 63, 1500, 2, 100, 3, 3], [130, 5, 1030, 5, 128, 5, 300, 5]], ids=str)
def test_short_rows_between_long_ones(seq, n_sm):
    """The route of three kernels: the split walks over the rows that the short kernel takes."""
    c = synthetic.make_layer_case(17, seq, "beta:2,5", 5e5, torch.bfloat16, "cpu", n_q_heads=8, n_kv_heads=2)
    a, out, ref, status = _run(c, _lib.load().dkv_routed_decode, n_sm, switch=64)
    assert _lib.load().dkv_routed_launches(ctypes.byref(a), 64) == 3
    assert status == 0 and float(_row_errors(out, ref).max()) <= _row_limit(torch.bfloat16)


def _raw_call(q, k_up, v_up, flat, lens, offs, stride):
    """dkv_two_stage_decode with K and V rows in one arena that is said to be `stride` elements wide."""
    out = torch.full(q.shape, 7.0, dtype=q.dtype, device="cuda")
    a, keep = _common.build_attn_args(q, flat, k_up, flat, v_up, lens, offs, lens, offs, 5e5, out=out, len_multiple=8, need_workspace=True)
    a.k.flat_stride = a.v.flat_stride = stride
    _lib.check(_lib.load().dkv_two_stage_decode(ctypes.byref(a)), "dkv_two_stage_decode")
    torch.cuda.synchronize()
    del keep
    return out, _common.read_status(torch.device("cuda"))


def _one_arena():
    c = synthetic.make_layer_case(23, [300], "uniform", 5e5, torch.bfloat16, "cuda", n_q_heads=4, n_kv_heads=1)
    gen = torch.Generator().manual_seed(23)
    lens = torch.randint(1, 17, (1, 300), generator=gen, dtype=torch.int32) * 8
    lens[0, -1] = 128
    side = synthetic.ragged_side(lens.cuda(), torch.Generator("cuda").manual_seed(23), torch.bfloat16)
    return (c.q, c.k_up, c.v_up), side.flat, side.lens[:, :300], side.offs[:, :300], int(lens.sum())


@pytest.mark.parametrize("end", [2 ** 31 - 8, 2 ** 31, 2 ** 31 + 120])
def test_arena_of_more_than_2_31_elements(end):
    """A row may end behind the largest int, as long as its arena goes on: the same result as from an arena of its own."""
    head, small, lens, offs, n = _one_arena()
    want, status = _raw_call(*head, small, lens, offs, n)
    assert status == 0
    flat = torch.empty(1, end, dtype=torch.bfloat16, device="cuda")
    shift = end - n
    flat[0, shift:] = small[0, :n]
    assert int(offs.max()) + shift <= 2 ** 31 - 1
    got, status = _raw_call(*head, flat, lens, offs + shift, end)
    assert status == 0 and torch.equal(got, want)
    cut, status = _raw_call(*head, flat, lens, offs + shift, end - 8)      # the last row does not fit
    assert status == 2 and not torch.equal(cut, want)


def test_arena_of_negative_size_holds_nothing():
    head, flat, lens, offs, _ = _one_arena()
    out, status = _raw_call(*head, flat, lens, offs, -8)
    assert status == 6 and float(out.abs().max()) == 0


def test_probe_of_the_tensor_pipe():
    """Every form ends in time; 8 x (M128 N128 K16) cannot take less than 512 cycles (4096 multiply-adds a cycle and SM)."""
    n, tiles, dev = 4, 50, torch.device("cuda")
    word = _common.status_word(dev)
    for mask, warps in ((1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (6, 1), (7, 1), (11, 2), (23, 1), (39, 1), (43, 2), (71, 3), (103, 3)):
        cyc = torch.zeros(3, n, dtype=torch.int64, device=dev)
        _lib.check(_lib.load().dkv_probe_tensor_pipe(mask, tiles, n, cyc.data_ptr(), word.data_ptr(), _lib.stream_ptr(dev)), "dkv_probe_tensor_pipe")
        assert _common.read_status(dev) == 0
        assert bool((cyc[:warps] > 0).all()) and not cyc[warps:].any()
        if mask & 1:
            assert float(cyc[0].min()) >= 0.98 * 512 * tiles
    assert _lib.load().dkv_probe_tensor_pipe(8, tiles, n, cyc.data_ptr(), word.data_ptr(), _lib.stream_ptr(dev)) != 0
