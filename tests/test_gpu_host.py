"""The native host side takes the calls that the Python side took: numbers of any kind, refusals and fallbacks alike."""
import pytest
import torch

from dynakv_b200 import synthetic
from dynakv_b200.kernels import _common
from dynakv_b200.kernels.compressed_cache import CustomDynamicCache
from dynakv_b200.kernels.fused import fused_attention_dispatch
from dynakv_b200.kernels.two_stage import abx_sparse, avx, two_stage_attention

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_numbers_of_any_kind():
    from dynakv_b200.kernels.compressed_attention import gate_lengths, kv_process_fused
    gen = torch.Generator().manual_seed(1)
    x, w, b = torch.randn(1, 5, 64, generator=gen).to(DEV), torch.randn(64, 64, generator=gen).to(DEV), torch.randn(64, generator=gen).to(DEV)
    masked, lens = gate_lengths(x, w, b, 48, len_multiple=8)
    for rank, yes, step in ((48.0, 1, 8.0), (torch.tensor(48), [0], 8), (torch.tensor(48.0), True, torch.tensor(8))):
        got, n = gate_lengths(x, w, b, rank, return_masked=yes, len_multiple=step)
        assert torch.equal(got, masked) and torch.equal(n, lens)
        assert torch.equal(kv_process_fused(x, x, w, b, w, b, rank, len_multiple=step)[2], lens)
    assert gate_lengths(x, w, b, 48, return_masked=0)[0] is None
    seq = [100, 700]
    c = synthetic.make_layer_case(5, seq, "beta:2,5", 5e5, torch.bfloat16, DEV)
    fk, fv, lk, lv, ok, ov = c.views()
    args = (c.q, fk, c.k_up, fv, c.v_up, lk, ok, lv, ov)
    rows = torch.tensor(seq, dtype=torch.int32, device=DEV)
    for fn in (fused_attention_dispatch, two_stage_attention):
        want = fn(*args, 5e5, seq_lens=rows, len_multiple=8, route_max_tokens=800)
        got = fn(*args, torch.tensor(5e5), seq_lens=rows, len_multiple=8.0, route_min_tokens=0.0, route_max_tokens=torch.tensor(800.0))
        assert torch.equal(got, want)
    assert _common.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("arenas,shape,taken", [(1, (3, 1), True), (1, (3,), True), (1, (3, 1, 1), True), (2, (3, 2, 1), True), (2, (3, 2), False),
                                                (2, (6,), False)], ids=str)
def test_lengths_of_a_new_token(arenas, shape, taken):
    cache = CustomDynamicCache(arenas_per_batch=arenas, len_multiple=8)
    x = torch.randn(3, 4, arenas * 128, device=DEV).bfloat16()
    lens = torch.full((3, arenas, 4), 8, dtype=torch.int32, device=DEV)
    cache.reserve(0, 3, 1024, 64, torch.bfloat16, DEV)
    cache.update_sp(x, lens, x, lens, arenas * 128, 0, 128)
    new, one = x[:, :1].contiguous(), torch.full(shape, 16, dtype=torch.int32, device=DEV)
    if taken:
        cache.update_sp(new, one, new, one, arenas * 128, 0, 128)
    else:
        with pytest.raises((RuntimeError, ValueError)):
            cache.update_sp(new, one, new, one, arenas * 128, 0, 128)
    assert cache.get_seq_length(0) == 4 + taken and cache.key_cache_sp[0][3].tolist() == [32 + 16 * taken] * 3 * arenas
    assert _common.read_status(torch.device(DEV)) == 0


def test_buffers_that_a_two_dimensional_copy_cannot_grow():
    n = 64
    one = torch.arange(n, device=DEV, dtype=torch.float32).bfloat16()
    odd = one.as_strided((1, n), (1, 1))              # one row: its stride says nothing
    ints = torch.zeros(1, 8, dtype=torch.int32, device=DEV)
    cache = CustomDynamicCache(len_multiple=8)
    cache.adopt(0, (odd, ints.clone(), ints.clone(), ints[:, 0].clone()), (odd.clone(), ints.clone(), ints.clone(), ints[:, 0].clone()), [0])
    x = torch.randn(1, 4, 128, device=DEV).bfloat16()
    lens = torch.full((1, 4), 64, dtype=torch.int32, device=DEV)
    cache.update_sp(x, lens, x, lens, 128, 0, 128, token_counts=[4])
    for state in (cache.key_cache_sp[0], cache.value_cache_sp[0]):
        assert state[3].tolist() == [256] and torch.equal(state[0][0, :256], x[0, :, :64].reshape(-1))
    big = torch.zeros(2, (1 << 30) - 8, dtype=torch.bfloat16, device=DEV)     # rows of 2 GiB less 16 bytes
    big[:, -1] = 3.0
    grown = CustomDynamicCache._grown(big, (1 << 30) + 8)
    assert grown.shape == (2, (1 << 30) + 8) and grown[:, (1 << 30) - 9].tolist() == [3.0, 3.0] and int(grown.count_nonzero()) == 2
    assert _common.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("tokens", [1, 20, 90, 700])
def test_operators_give_what_the_general_path_gives(tokens, dtype):
    # a basis that records gradients, strided queries and scores, lengths as columns of a wider buffer, a heads axis of one
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    B, R, A = 2, 96, 2
    lens = torch.randint(1, R + 1, (B * A, tokens + 5), generator=gen, device=DEV, dtype=torch.int32)
    offs = (torch.cumsum(lens, 1) - lens).to(torch.int32)
    flat = torch.randn(B * A, int(lens.sum(1).max()), generator=gen, device=DEV).to(dtype)
    up = (torch.randn(4, R, 128, generator=gen, device=DEV) / R ** 0.5).to(dtype)
    q = torch.randn(B, 8, 256, generator=gen, device=DEV).to(dtype)[:, :, ::2]
    lens, offs = lens[:, :tokens], offs[:, :tokens]
    want = abx_sparse(q.contiguous(), up, flat, lens, offsets=offs, theta=5e5)
    general = abx_sparse(q.contiguous(), up.clone().requires_grad_(), flat, lens, offsets=offs, theta=5e5)
    assert torch.equal(want, general) and torch.equal(want, abx_sparse(q, up, flat, lens.view(B, A, -1), offsets=offs.view(B, A, -1), theta=5e5))
    out = avx(want, flat, up, lens, offs)
    wide = torch.zeros(B, 8, 2 * tokens, dtype=dtype, device=DEV)
    wide[:, :, ::2] = want
    for got in (avx(want, flat, up.clone().requires_grad_(), lens, offs), avx(want.unsqueeze(2), flat.view(B, A, -1), up, lens, offs),
                avx(wide[:, :, ::2], flat, up, lens, offs)):
        assert torch.equal(got, out)
    assert _common.read_status(torch.device(DEV)) == 0
