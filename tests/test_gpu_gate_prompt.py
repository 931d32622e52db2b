"""The gate over many 16-bit rows (tensor-core logits): edges of the 128-row tiles, every width it takes, padded rows."""
import pytest
import torch

from oracle import dynakv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("rows,d,low_rank,pad", [(65, 128, 128, 0), (128, 256, 200, 8), (129, 512, 512, 0), (300, 1024, 640, 64),
                                                 (4800, 1024, 1024, 0)])
def test_gate_of_a_prompt_against_oracle(rows, d, low_rank, pad, dtype):
    from dynakv_b200.kernels.compressed_attention import gate_lengths
    gen = torch.Generator().manual_seed(rows + d)
    wide = (torch.randn(rows, d + pad, generator=gen) * 2).to(dtype)
    x = wide[:, :d]
    W = (torch.randn(d, d, generator=gen) / d ** 0.5).to(dtype)
    b = (torch.randn(d, generator=gen) * 0.5).to(dtype)
    ref = O.gate_lengths(x.float(), W.float(), b.float(), low_rank).to(torch.int64)
    masked, lens = gate_lengths(wide.cuda()[:, :d], W.cuda(), b.cuda(), low_rank, native_rounding=False)
    diff = lens.cpu().to(torch.int64) - ref
    assert int(diff.abs().max()) <= 1 and int((diff != 0).sum()) <= 1 + rows // 500     # summation order only
    keep = torch.arange(d)[None, :] < lens.cpu()[:, None]
    assert torch.equal(masked.cpu(), torch.where(keep, x, torch.zeros_like(x)))
    _, lens8 = gate_lengths(wide.cuda()[:, :d], W.cuda(), b.cuda(), low_rank, native_rounding=False, len_multiple=8, return_masked=False)
    assert torch.equal(lens8, torch.clamp((lens + 7) // 8 * 8, max=d))


@pytest.mark.parametrize("rows,d", [(70, 128), (1000, 512), (3000, 1024)])
def test_both_sides_in_one_launch_give_what_each_gives(rows, d):
    from dynakv_b200.kernels.compressed_attention import gate_lengths, kv_process_fused
    gen = torch.Generator().manual_seed(rows)
    side = lambda: (torch.randn(2, rows // 2, d, generator=gen).bfloat16().cuda(), (torch.randn(d, d, generator=gen) / d ** 0.5).bfloat16().cuda(),
                    torch.randn(1, d, generator=gen).bfloat16().cuda())
    (k, wk, bk), (v, wv, bv) = side(), side()
    k_out, v_out, len_k, len_v, _, _ = kv_process_fused(k, v, wk, bk, wv, bv, d)
    for (out, lens), got in ((gate_lengths(k, wk, bk, d), (k_out, len_k)), (gate_lengths(v, wv, bv, d), (v_out, len_v))):
        assert torch.equal(out, got[0]) and torch.equal(lens, got[1])


def test_the_gate_reports_to_the_status_word(monkeypatch):
    # a wait that runs out cannot be had without a broken kernel: what is checked is where the calls would report it
    from dynakv_b200 import _lib
    from dynakv_b200.kernels import _common
    from dynakv_b200.kernels.compressed_attention import gate_lengths, gate_lengths_pair, kv_process_fused
    dev = torch.device("cuda")
    word, seen, lib = _common.status_word(dev).data_ptr(), [], _lib.load()
    for name in ("dkv_gate_lengths", "dkv_gate_lengths_pair"):
        real = getattr(lib, name)
        monkeypatch.setattr(lib, name, lambda *a, real=real: (seen.extend(x._obj.status for x in a), real(*a))[1])
    x, w, b = torch.randn(200, 128, device=dev).bfloat16(), torch.randn(128, 128, device=dev).bfloat16(), torch.zeros(128, device=dev).bfloat16()
    lens = torch.empty(200, dtype=torch.int32, device=dev)
    gate_lengths(x, w, b, 128, out_lengths=lens)
    gate_lengths_pair(x, w, b, x, w, b, 128, lens, lens.clone())
    assert seen == [word] * 3
    gate_lengths(x, w, b, 128)
    kv_process_fused(x[None], x[None], w, b, w, b, 128)
    assert _common.read_status(dev) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("rows", [64, 65, 512])
def test_pair_and_prompt_paths_differ_by_summation_order_only(rows, dtype):
    # dkv_gate_lengths takes more than 64 16-bit rows of 128 from the tensor core, the pair adds up in ascending order
    from dynakv_b200.kernels.compressed_attention import gate_lengths, gate_lengths_pair
    gen, d, thr = torch.Generator().manual_seed(rows), 128, 0.1
    x, v = ((torch.randn(rows, d, generator=gen) * 2).to(dtype).cuda() for _ in range(2))
    w, b = (torch.randn(d, d, generator=gen) / d ** 0.5).to(dtype).cuda(), (torch.randn(d, generator=gen) * 0.5).to(dtype).cuda()
    lk, lv = (torch.empty(rows, dtype=torch.int32, device="cuda") for _ in range(2))
    gate_lengths_pair(x, w, b, v, w, b, d, lk, lv, native_rounding=False)
    for states, pair in ((x, lk), (v, lv)):
        _, lens = gate_lengths(states, w, b, d, native_rounding=False)
        if rows <= 64 or dtype == torch.float32:
            assert torch.equal(lens, pair)
            continue
        logits = states.double() @ w.double() + b.double()
        sums = torch.cumsum(torch.softmax(logits, -1), -1)
        # a logit is a sum of 129 terms: off by at most 129 units of 2^-23 of the terms' sum (2^-24 if rounded, twice that if cut);
        # a probability by twice the largest of these, relative, and a running sum of them by as much of itself and 256 roundings
        off = 129 * 2.0 ** -23 * (states.double().abs() @ w.double().abs() + b.double().abs()).amax(-1, keepdim=True)
        tie = (sums - thr).abs() <= sums * (2 * off + 256 * 2.0 ** -23)
        differ = lens != pair
        assert bool(tie.any(-1)[differ].all()) and int((lens - pair).abs().max()) <= int(tie.sum(-1).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("d", [128, 1024])
@pytest.mark.parametrize("thr", [0.1, 0.5, 0.50390625, 0.7529296875, 0.998046875, 1.0, 1.5, 0.0, -1.0, 1e-30, float("inf"), float("nan")])
def test_bound_of_rounded_sums(thr, d, native, dtype):
    """Equal logits: probabilities 1/d and sums j/d are exact, and for d = 1024 their roundings are not: ties on both sides."""
    from dynakv_b200.kernels.compressed_attention import gate_lengths
    rows = 65
    x = torch.randn(rows, d, device="cuda").to(dtype)
    w, b = torch.zeros(d, d, device="cuda", dtype=dtype), torch.full((d,), 0.5, device="cuda", dtype=dtype)
    sums = torch.arange(1, d + 1, dtype=torch.float32) / d
    bound = torch.tensor(thr, dtype=torch.float32)
    if native:
        sums, bound = sums.to(dtype).float(), bound.to(dtype).float()
    for low_rank in (d, d - 37):
        want = int((sums[d - low_rank:] >= bound).sum())
        got = gate_lengths(x, w, b, low_rank, threshold=thr, return_masked=False, native_rounding=native)[1]
        assert got.cpu().tolist() == [want] * rows


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("d", [128, 256, 512, 1024])
@pytest.mark.parametrize("thr", [0.1, 0.6, 0.97])
def test_lengths_of_unequal_logits(thr, d, native, dtype):
    """Identity weights: a row's logits are its own elements, spread by 0.5 to 120.  The lengths are those of 64-bit sums of the
    softmax, with the roundings to the storage type that `native` asks for, except where a sum ties with the threshold."""
    from dynakv_b200.kernels.compressed_attention import gate_lengths
    rows = 600
    gen = torch.Generator().manual_seed(d)
    spread = torch.tensor([0.5, 3.0, 10.0, 40.0, 120.0]).repeat(rows // 5)[:, None]
    x = (-torch.rand(rows, d, generator=gen) * spread).to(dtype)
    got = gate_lengths(x.cuda(), torch.eye(d, dtype=dtype, device="cuda"), torch.zeros(d, dtype=dtype, device="cuda"), d, threshold=thr,
                       return_masked=False, native_rounding=native)[1].cpu().long()
    p = torch.softmax(x.double(), -1)
    # relative error of a probability, and of a sum of them: 2 units of the exponential, 30 / 2 of its argument (smaller ones do not
    # count), a half for each of the 37 additions of the sum, the quotient and another 37: below 64 units of 2^-23
    err = 64 * 2.0 ** -23
    slack = torch.zeros(rows, 1, dtype=torch.float64)
    bound = float(torch.tensor(thr, dtype=torch.float32))
    if native:
        digits, least = (8, -133) if dtype == torch.bfloat16 else (11, -24)
        ulp = torch.ldexp(torch.ones_like(p), (torch.frexp(p).exponent - digits).clamp_min(least))
        near = ((p / ulp - torch.floor(p / ulp) - 0.5).abs() <= err * p / ulp)      # may be rounded to either side
        slack = (near * ulp).cumsum(-1)
        p = p.to(dtype).double()
        bound = float(torch.tensor(thr, dtype=dtype))
    sums = p.cumsum(-1)
    lo, hi = sums * (1 - err) - slack, sums * (1 + err) + slack
    if native:
        lo, hi = lo.to(dtype).double(), hi.to(dtype).double()
    least, most = (lo >= bound).sum(-1), (hi >= bound).sum(-1)
    assert bool(((least <= got) & (got <= most)).all())
    assert float((most > least).double().mean()) <= 0.1        # ties are few: nearly every row is held to one length
