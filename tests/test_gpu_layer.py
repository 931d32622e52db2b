"""Row operators of a decode step against the torch chains that they stand for: rows and columns that are no multiples of
the thread counts, one row, ties of the maximum."""
import pytest
import torch
import torch.nn.functional as F

from dynakv_b200 import runner, synthetic

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])


def _close(a, b, dtype):
    tol = {torch.float32: 1e-6, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dtype]       # one rounding
    assert torch.allclose(a.float(), b.float(), rtol=tol, atol=tol * 1e-2)


@DTYPES
@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 515), (5, 4096), (2, 13000)])
def test_norm_and_cutoffs(rows, dim, dtype):
    gen = torch.Generator().manual_seed(dim)
    h, y = (torch.randn(rows, dim, generator=gen).to(dtype).cuda() for _ in range(2))
    w = (1.0 + 0.1 * torch.randn(dim, generator=gen)).to(dtype).cuda()
    w_cut = (torch.randn(6, dim, generator=gen) / dim ** 0.5).cuda()
    h1, h2 = h.clone(), h + y
    x, none, _ = runner._norm_rows(h1, None, w, 1e-5)
    assert none is None and torch.equal(h1, h)
    _close(x, runner.rms_norm(h, w, 1e-5), dtype)
    x, lk, lv = runner._norm_rows(h1, y, w, 1e-5, w_cut, -0.5)
    assert torch.equal(h1, h2)
    _close(x, runner.rms_norm(h2, w, 1e-5), dtype)
    want = synthetic.cutoff_head_lengths(x, w_cut, -0.5)
    assert int((torch.cat((lk, lv), 1) - want).abs().max()) <= 8 and torch.cat((lk, lv), 1).eq(want).float().mean() > 0.8   # sums in another order


@DTYPES
@pytest.mark.parametrize("rows,n_q,n_kv", [(1, 4, 1), (3, 6, 2), (2, 32, 8)])
def test_split_qkv(rows, n_q, n_kv, dtype):
    qkv = torch.randn(rows, (n_q + 2 * n_kv) * 128, generator=torch.Generator().manual_seed(rows)).to(dtype).cuda()
    pos = torch.tensor([0, 31000, 7][:rows], dtype=torch.int32, device="cuda")
    q, k, v = runner._split_qkv(qkv, n_q, n_kv, pos, 5e5)
    wq, wk, wv = (t.reshape(rows, -1, 128) for t in qkv.split((n_q * 128, n_kv * 128, n_kv * 128), dim=1))
    assert torch.equal(k, wk) and torch.equal(v, wv)
    assert float((q.float() - runner.rope(wq, pos, 5e5).float()).abs().max()) <= {torch.float32: 1e-4}.get(dtype, 3e-2)


@DTYPES
@pytest.mark.parametrize("rows,n", [(1, 1), (3, 517), (2, 14336), (4, 32001)])
def test_silu_and_argmax(rows, n, dtype):
    gu = torch.randn(rows, 2 * n, generator=torch.Generator().manual_seed(n)).to(dtype).cuda()
    _close(runner._silu_mul(gu), F.silu(gu[:, :n]) * gu[:, n:], dtype)
    x = gu[:, :n]           # 16-bit rows of odd lengths start off a 16-byte boundary; few values, so many ties
    assert torch.equal(runner._argmax_rows(x).cpu(), torch.tensor([int((r == r.max()).nonzero()[0]) for r in x.float().cpu()]))


def test_argmax_of_more_clusters_than_the_gpu_holds():
    # 1500 rows x 4 CTAs: the CTAs of a cluster start while others of the launch still run
    x = torch.randint(-50, 50, (1500, 30000), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    x[torch.arange(1500), torch.arange(1500) * 19 % 30000] = 60.0
    for _ in range(3):
        assert torch.equal(runner._argmax_rows(x).cpu(), torch.arange(1500) * 19 % 30000)
