"""Blocks of tokens packed into a layer and expanded again: pieces that are not 16-byte aligned, rows that are no whole
number of pieces, growth behind a block that did not fit at first, ragged counts."""
import numpy as np
import pytest
import torch

from dynakv_b200.kernels import _common
from dynakv_b200.kernels.compressed_cache import CustomDynamicCache
from oracle import dynakv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,step,dtype", [(128, 8, torch.bfloat16), (128, 1, torch.float16), (100, 1, torch.float32), (12, 4, torch.bfloat16)])
def test_blocks_grow_and_expand_like_the_layout_oracle(R, step, dtype):
    gen = torch.Generator().manual_seed(R + step)
    B, A = 2, 3
    cache = CustomDynamicCache(arenas_per_batch=A, len_multiple=step)
    cache.reserve(0, B, 8 * R, 64, dtype, "cuda")           # the second block does not fit: the buffers grow behind it
    lays = [O.LayoutOracle(B * A, np.float32) for _ in range(2)]
    for n_new, counts in ((5, None), (37, None), (1, None), (300, None), (4200, None)):
        rows = [torch.randn(B, n_new, A * R, generator=gen).to(dtype) for _ in range(2)]
        lens = [(torch.randint(0, R // step + 1, (B, A, n_new), generator=gen) * step).to(torch.int32) for _ in range(2)]
        cache.update_sp(rows[0].cuda(), lens[0].cuda(), rows[1].cuda(), lens[1].cuda(), A * R, 0, R, token_counts=counts)
        for lay, x, n in zip(lays, rows, lens):
            lay.update(x.float().view(B, n_new, A, R).permute(0, 2, 1, 3).reshape(B * A, n_new, R).numpy(), n.view(B * A, n_new).numpy())
    for lay, state, dense in zip(lays, (cache.key_cache_sp[0], cache.value_cache_sp[0]), cache.get_origin_states(R, 0)):
        s = state[4]
        assert np.array_equal(state[1][:, :s].cpu().numpy(), lay.lens) and np.array_equal(state[3].cpu().numpy(), lay.ptr)
        assert state[5] == [int(x) for x in lay.ptr]
        for r in range(B * A):
            assert np.array_equal(state[0][r, : lay.ptr[r]].float().cpu().numpy(), lay.flat[r])
            want = np.zeros((s, R), np.float32)
            for t in range(s):
                want[t, : lay.lens[r, t]] = lay.flat[r][lay.offs[r, t]: lay.offs[r, t] + lay.lens[r, t]]
            assert np.array_equal(dense[r].float().cpu().numpy(), want)
    assert _common.read_status(torch.device("cuda")) == 0


def test_ragged_block_keeps_each_rows_count():
    B, A, R, S = 2, 2, 128, 20
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(B, S, A * R, generator=gen).to(torch.bfloat16).cuda()
    lens = (torch.randint(1, 17, (B, A, S), generator=gen) * 8).to(torch.int32)
    cache = CustomDynamicCache(arenas_per_batch=A, len_multiple=8)
    cache.update_sp(x, lens.cuda(), x, lens.cuda(), A * R, 0, R, token_counts=[7, S])
    assert cache.seq_lens(0).tolist() == [7, S] and cache.seq_lens_host(0) == [7, S]
    stored = torch.stack([lens[0, :, :7].sum(1), lens[1].sum(1)]).view(-1)
    assert cache.key_cache_sp[0][3].tolist() == stored.tolist() == cache.key_cache_sp[0][5]
    assert _common.read_status(torch.device("cuda")) == 0
