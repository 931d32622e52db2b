"""Tile kernels (any layout with a workspace): tile and slice edges, odd ranks, one and many heads per group or arena,
rows that start at any element, bases that are not 16-byte aligned."""
import pytest
import torch

from dynakv_b200.kernels import _common
from dynakv_b200.kernels.fused import fused_attention_dispatch
from dynakv_b200.kernels.two_stage import abx_sparse, avx, two_stage_attention
from oracle import dynakv_oracle as O

pytestmark = pytest.mark.gpu


def _case(seed, B, S, R, Hq, groups, arenas, dtype):
    gen = torch.Generator().manual_seed(seed)
    t = {"q": torch.randn(B, Hq, 128, generator=gen).to(dtype)}
    for side in "kv":
        lens = torch.randint(0, R + 1, (B * arenas, S), generator=gen, dtype=torch.int32)
        lens[:, 0].clamp_(min=1)
        offs = (torch.cumsum(lens.long(), 1) - lens.long()).to(torch.int32)
        cap = int(lens.long().sum(1).max()) + 3
        sigma = torch.exp(-torch.arange(R, dtype=torch.float32) / max(R / 4, 1))
        t["flat_" + side] = (torch.randn(B * arenas, cap, generator=gen) * sigma[torch.arange(cap) % R]).to(dtype)
        t["lens_" + side], t["offs_" + side] = lens, offs
        t[side + "_up"] = (torch.randn(groups, R, 128, generator=gen) / R ** 0.5).to(dtype)
    return t


def _dev(t, shift):
    d = {k: v.cuda() for k, v in t.items()}
    if shift:       # bases that start two bytes past a 16-byte boundary
        for k in ("k_up", "v_up"):
            buf = torch.empty(d[k].numel() + 1, dtype=d[k].dtype, device="cuda")
            buf[1:].copy_(d[k].view(-1))
            d[k] = buf[1:].view(d[k].shape)
    return d


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("B,S,R,Hq,groups,arenas,shift", [
    (1, 1, 8, 4, 1, 1, 0), (2, 127, 63, 8, 2, 2, 0), (1, 129, 64, 12, 1, 1, 1), (3, 33, 819, 32, 8, 1, 0), (1, 300, 1024, 40, 40, 1, 0),
    (1, 130, 513, 36, 4, 1, 1),
    # around the lines below which the operators take one kernel (32 tokens; 64 for the fp32 softmax; 592 rows x heads)
    (2, 32, 256, 32, 8, 1, 0), (1, 64, 100, 16, 4, 4, 0), (1, 65, 40, 16, 16, 2, 0), (19, 32, 72, 32, 8, 1, 0), (18, 31, 72, 32, 32, 1, 1),
    # one basis for several arenas, basis groups that straddle arenas
    (2, 70, 24, 8, 1, 4, 0), (1, 150, 100, 12, 2, 3, 0), (2, 129, 64, 24, 4, 3, 1), (1, 260, 128, 32, 2, 32, 0)])
def test_tile_kernels_against_oracle(B, S, R, Hq, groups, arenas, shift, dtype):
    t = _case(S + R, B, S, R, Hq, groups, arenas, dtype)
    d = _dev(t, shift)
    knw = 1.0 + 0.1 * torch.randn(128, generator=torch.Generator().manual_seed(1)) if S == 33 else None
    ref = O.compact_attention(*(t[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")), 10000.0,
                              k_norm_weight=knw)
    args = [d[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")]
    kw = {} if knw is None else dict(k_norm_weight=knw.cuda())
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for fn in (fused_attention_dispatch, two_stage_attention):
        out = fn(*args, 10000.0, **kw).float().cpu()
        assert float((out - ref).abs().max()) <= tol * max(1.0, float(ref.abs().max()))
    if knw is None:
        # the stage operators chained: scores in the query type, then the softmax over them
        sc = abx_sparse(d["q"], d["k_up"], d["flat_k"], d["lens_k"], offsets=d["offs_k"], theta=10000.0)
        out = avx(sc, d["flat_v"], d["v_up"], d["lens_v"], d["offs_v"]).float().cpu()
        loose = tol if dtype == torch.float32 else 4e-2
        assert float((out - ref).abs().max()) <= loose * max(1.0, float(ref.abs().max()))
    assert _common.read_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_ragged_rows_over_several_slices(dtype):
    # 9000 tokens: 64 slices of more than one tile, a short row whose other slices are empty, an empty row
    t = _case(5, 3, 9000, 24, 8, 2, 1, dtype)
    d = _dev(t, 0)
    seq = [9000, 150, 0]
    ref = O.compact_attention(*(t[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")), 500000.0,
                              seq_lens=seq)
    args = [d[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")]
    out = two_stage_attention(*args, 500000.0, seq_lens=torch.tensor(seq, dtype=torch.int32, device="cuda")).float().cpu()
    assert float((out - torch.nan_to_num(ref)).abs().max()) <= (2e-4 if dtype == torch.float32 else 2e-2)
    assert _common.read_status(torch.device("cuda")) == 4       # the empty row is reported


def test_softmax_operator_reads_the_counter_behind_an_append():
    # the append lets the kernel behind it start early and moves the rows' counters on at its end
    import ctypes as C

    from dynakv_b200 import _lib, synthetic
    from dynakv_b200.kernels._common import build_attn_args
    from dynakv_b200.kernels.compressed_attention import CompressedDecodeLayer
    from dynakv_b200.kernels.compressed_cache import CustomDynamicCache
    B, H, n, steps = 4, 8, 20, 12
    c = synthetic.make_layer_case(9, [n] * B, "beta:2,5", 5e5, torch.bfloat16, "cuda", extra_tokens=steps)
    cache = CustomDynamicCache(arenas_per_batch=H, len_multiple=8)
    cache.adopt(0, (c.k.flat, c.k.lens, c.k.offs, c.k.ptr), (c.v.flat, c.v.lens, c.v.offs, c.v.ptr), [n] * B)
    layer = CompressedDecodeLayer(0, c.k_up, c.v_up, 5e5, project_new_rows=True)
    layer.prepare(B, "cuda")
    flat, lens, offs = cache.value_cache_sp[0][:3]
    cap, counter = lens.shape[1], cache.seq_lens(0)
    gen = torch.Generator(device="cuda").manual_seed(2)
    scores = torch.arange(cap, device="cuda").float().expand(B, 32, cap).contiguous().bfloat16()      # the last token weighs most
    lengths = torch.full((B, H), 64, dtype=torch.int32, device="cuda")
    for step in range(1, steps + 1):
        new = torch.randn(B, H, 128, generator=gen, device="cuda").bfloat16()
        out = torch.empty(B, 32, 128, dtype=torch.bfloat16, device="cuda")
        args, keep = build_attn_args(None, None, None, flat, c.v_up, None, None, lens, offs, 1e4, out=out, seq_lens=counter, need_workspace=True)
        torch.cuda.synchronize()
        layer.append(cache, new, new, lengths, lengths, counter, cap)
        _lib.check(_lib.load().dkv_softmax_v(C.byref(args), scores.data_ptr(), scores.stride(0), scores.stride(1)), "dkv_softmax_v")
        del keep
        s = n + step
        ref = O.softmax_v_reference(scores[:, :, :s].float().cpu(), flat.float().cpu(), c.v_up.float().cpu(), lens[:, :s].cpu(), offs[:, :s].cpu())
        assert float((out.float().cpu() - ref).abs().max()) <= 2e-2 * max(1.0, float(ref.abs().max()))
    assert _common.read_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("poison", ["query", "key", "key_inf", "value"])
def test_what_is_not_finite_stays_so(poison, dtype):
    # 300 tokens, none of them empty: a NaN query leaves no score that is a number in any slice
    t = _case(3, 1, 300, 64, 8, 2, 1, dtype)
    for side in "kv":
        t["lens_" + side] = t["lens_" + side].clamp(min=1)
        t["offs_" + side] = (torch.cumsum(t["lens_" + side], 1) - t["lens_" + side]).to(torch.int32)
        t["flat_" + side] = torch.randn(1, int(t["lens_" + side].sum()), generator=torch.Generator().manual_seed(8)).to(dtype)
    where, at, value = {"query": ("q", (0, 3, 5), "nan"), "key": ("flat_k", (0, 40), "nan"), "key_inf": ("flat_k", (0, 40), "inf"),
                        "value": ("flat_v", (0, 0), "nan")}[poison]
    t[where][at] = float(value)
    want = torch.zeros(8, dtype=torch.bool)
    want[3 if poison == "query" else slice(None)] = True
    d = _dev(t, 0)
    args = [d[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")]
    outs = [fn(*args, 10000.0) for fn in (fused_attention_dispatch, two_stage_attention)]
    outs.append(avx(abx_sparse(d["q"], d["k_up"], d["flat_k"], d["lens_k"], offsets=d["offs_k"]), d["flat_v"], d["v_up"], d["lens_v"], d["offs_v"]))
    for out in outs:
        assert torch.equal(out[0].isnan().any(-1).cpu(), want)
    _common.read_status(torch.device("cuda"))


@pytest.mark.parametrize("longest", [1, 7, 15, 16, 17, 70])
@pytest.mark.parametrize("value", ["nan", "inf"])
def test_fp32_basis_rows_that_no_token_reaches_take_no_part(value, longest):
    t = _case(4, 1, 100, 96, 8, 2, 1, torch.float32)
    for side in "kv":
        t["lens_" + side] = t["lens_" + side].clamp(min=1, max=longest)
        t["offs_" + side] = (torch.cumsum(t["lens_" + side], 1) - t["lens_" + side]).to(torch.int32)
    outs = []
    for fill in (0.0, float(value)):
        t["k_up"][:, longest:] = fill
        d = _dev(t, 0)
        args = [d[k] for k in ("q", "flat_k", "k_up", "flat_v", "v_up", "lens_k", "offs_k", "lens_v", "offs_v")]
        outs.append([fn(*args, 10000.0) for fn in (fused_attention_dispatch, two_stage_attention)]
                    + [abx_sparse(d["q"], d["k_up"], d["flat_k"], d["lens_k"], offsets=d["offs_k"], theta=10000.0)])
    assert all(torch.equal(a, b) and bool(b.isfinite().all()) for a, b in zip(*outs))
    assert _common.read_status(torch.device("cuda")) == 0
