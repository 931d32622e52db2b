"""Short-cache fused kernel: tile and cluster edges (one to four CTAs, rows walked in several rounds), one to four query
heads per group, bases of fewer coefficients, rows of other lengths in the launch, rows without tokens."""
import pytest
import torch

from dynakv_b200 import synthetic
from dynakv_b200.kernels import _common
from dynakv_b200.kernels.fused import fused_attention_dispatch
from dynakv_b200.kernels.two_stage import two_stage_attention
from oracle import dynakv_oracle as O

pytestmark = pytest.mark.gpu


def _run(seq, dtype, hq, hkv, knorm=False, rank=128, shift=False, entry=fused_attention_dispatch):
    c = synthetic.make_layer_case(sum(seq) + hq, seq, "beta:2,5", 5e5, dtype, "cpu", n_q_heads=hq, n_kv_heads=hkv)
    fk, fv, lk, lv, ok, ov = c.views()
    k_up, v_up = c.k_up, c.v_up
    if rank < 128:
        lk, lv = lk.clamp(max=rank), lv.clamp(max=rank)
        k_up, v_up = k_up[:, :rank].contiguous(), v_up[:, :rank].contiguous()
    knw = 1.0 + 0.1 * torch.randn(128, generator=torch.Generator().manual_seed(1)) if knorm else None
    ref = O.compact_attention(c.q, fk, k_up, fv, v_up, lk, ok, lv, ov, c.theta, seq_lens=seq, k_norm_weight=knw)
    d = [t.cuda() for t in (c.q, fk, k_up, fv, v_up, lk, ok, lv, ov)]
    if shift:       # a V basis that starts two bytes past a 16-byte boundary
        buf = torch.empty(v_up.numel() + 1, dtype=dtype, device="cuda")
        buf[1:].copy_(v_up.cuda().view(-1))
        d[4] = buf[1:].view(v_up.shape)
    kw = {} if knw is None else dict(k_norm_weight=knw.cuda())
    out = entry(*d, c.theta, seq_lens=torch.tensor(seq, dtype=torch.int32, device="cuda"), len_multiple=8, **kw).float().cpu()
    assert float((out - torch.nan_to_num(ref)).abs().max()) <= 2e-2 * max(1.0, float(torch.nan_to_num(ref).abs().max()))
    assert _common.read_status(torch.device("cuda")) == (4 if 0 in seq else 0)      # an empty row is reported


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("seq", [[1], [127, 128], [129, 1, 256], [257, 384, 128, 0], [500, 385], [1100, 512, 513, 3]], ids=str)
def test_tile_and_cluster_edges(seq, dtype):
    _run(seq, dtype, 32, 8, knorm=len(seq) == 3)


@pytest.mark.parametrize("hq,rank,shift", [(2, 128, False), (4, 64, False), (6, 40, True), (8, 128, True)])
def test_heads_per_group_and_bases(hq, rank, shift):
    _run([300, 70], torch.bfloat16, hq, 2, rank=rank, shift=shift)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("rows,rank", [(18, 128), (19, 128), (40, 120)])
def test_shifted_bases_on_both_sides_of_the_split(rows, rank, dtype):
    # 8 KV heads, 300 tokens: one kernel up to 148 (row, head) pairs, split and merge past them
    _run([300, 140] * (rows // 2) + [1] * (rows % 2), dtype, 32, 8, rank=rank, shift=True)


def test_shifted_bases_of_one_long_row():
    _run([3000], torch.bfloat16, 8, 2, shift=True, entry=two_stage_attention)


def test_one_tile_rows_of_more_ctas_than_the_gpu_holds():
    _run([128] * 150 + [5] * 50, torch.bfloat16, 16, 4)


@pytest.mark.parametrize("seq", [[1, 130, 499, 500, 640] * 8, [256] * 40], ids=["straddling", "short"])
def test_batches_whose_rows_go_through_the_split(seq):
    # 40 rows x 8 KV heads of more than one tile: past the line where the fused entry becomes split and merge
    from dynakv_b200.kernels.router import compressed_decode_attention
    c = synthetic.make_layer_case(5, seq, "beta:2,5", 5e5, torch.bfloat16, "cpu")
    fk, fv, lk, lv, ok, ov = c.views()
    ref = O.compact_attention(c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov, c.theta, seq_lens=seq)
    d = [t.cuda() for t in (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)]
    lens = torch.tensor(seq, dtype=torch.int32, device="cuda")
    outs = [fused_attention_dispatch(*d, c.theta, seq_lens=lens, len_multiple=8)]
    outs.append(compressed_decode_attention(q=d[0], k_flat=d[1], k_up=d[2], v_flat=d[3], v_up=d[4], key_lengths=d[5], key_offsets=d[6],
                                            value_lengths=d[7], value_offsets=d[8], theta=c.theta, cache_length=max(seq), seq_lens=lens,
                                            len_multiple=8))
    for out in outs:
        assert float((out.float().cpu() - ref).abs().max()) <= 2e-2
    assert _common.read_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("bounds", [dict(route_min_tokens=200), dict(route_max_tokens=200), dict(route_min_tokens=100, route_max_tokens=300)],
                         ids=["min", "max", "both"])
@pytest.mark.parametrize("rows", [2, 16, 24])
def test_rows_out_of_bounds_are_left_alone(rows, bounds):
    # 499 columns, 8 KV heads: the short kernel's cluster, the pipeline of one CTA per row, split and merge
    seq = [(0, 60, 199, 200, 299, 300, 499)[i % 7] for i in range(rows)]
    c = synthetic.make_layer_case(7, seq, "beta:2,5", 5e5, torch.bfloat16, "cpu")
    fk, fv, lk, lv, ok, ov = c.views()
    ref = O.compact_attention(c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov, c.theta, seq_lens=seq)
    out = torch.full(c.q.shape, 7.0, dtype=torch.bfloat16, device="cuda")
    fused_attention_dispatch(*(t.cuda() for t in (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)), c.theta, out=out, len_multiple=8,
                             seq_lens=torch.tensor(seq, dtype=torch.int32, device="cuda"), **bounds)
    lo, hi = bounds.get("route_min_tokens", 0), bounds.get("route_max_tokens", 1 << 30)
    for b, n in enumerate(seq):
        if lo <= n < hi:
            assert float((out[b].float().cpu() - torch.nan_to_num(ref[b])).abs().max()) <= 2e-2
        else:
            assert bool((out[b] == 7.0).all())
    assert _common.read_status(torch.device("cuda")) == (4 if lo == 0 and 0 in seq else 0)      # only a row that takes part is reported


@pytest.mark.parametrize("switch", [0, -1, 1])
@pytest.mark.parametrize("mult", [8, 1], ids=["packed", "any_length"])
def test_router_whose_policy_makes_every_row_long(switch, mult):
    from dynakv_b200.kernels.router import KernelPolicy, compressed_decode_attention
    seq = [100, 700, 1]
    c = synthetic.make_layer_case(11, seq, "beta:2,5", 5e5, torch.bfloat16, "cpu")
    fk, fv, lk, lv, ok, ov = c.views()
    ref = O.compact_attention(c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov, c.theta, seq_lens=seq)
    d = [t.cuda() for t in (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)]
    out = compressed_decode_attention(q=d[0], k_flat=d[1], k_up=d[2], v_flat=d[3], v_up=d[4], key_lengths=d[5], key_offsets=d[6],
                                      value_lengths=d[7], value_offsets=d[8], theta=c.theta, cache_length=700, len_multiple=mult,
                                      seq_lens=torch.tensor(seq, dtype=torch.int32, device="cuda"), policy=KernelPolicy(switch_tokens=switch))
    assert float((out.float().cpu() - ref).abs().max()) <= 2e-2
    assert _common.read_status(torch.device("cuda")) == 0
