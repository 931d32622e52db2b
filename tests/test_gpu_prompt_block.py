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


@pytest.mark.parametrize("k_type,v_type,k_dim,v_dim", [(torch.bfloat16, torch.float16, 128, 128), (torch.float32, torch.bfloat16, 128, 128),
                                                       (torch.bfloat16, torch.bfloat16, 64, 128), (torch.float16, torch.float16, 128, 72)])
def test_sides_of_other_types_and_widths(k_type, v_type, k_dim, v_dim):
    # a fresh layer, a block that fits and one that grows it; the joint layout's row width is the keys'
    gen = torch.Generator().manual_seed(k_dim + v_dim)
    B, width = 2, min(k_dim, v_dim)
    cache = CustomDynamicCache(len_multiple=8)
    types, lays = (k_type, v_type), [O.LayoutOracle(B, np.float32) for _ in range(2)]
    for n_new in (9, 3, 200):
        rows = [torch.randn(B, n_new, d, generator=gen).to(t) for d, t in zip((k_dim, v_dim), types)]
        lens = [(torch.randint(0, width // 8 + 1, (B, n_new), generator=gen) * 8).to(torch.int32) for _ in range(2)]
        cache.update_sp(rows[0].cuda(), lens[0].cuda(), rows[1].cuda(), lens[1].cuda(), k_dim, 0, k_dim)
        for lay, x, n in zip(lays, rows, lens):
            lay.update(x[:, :, :width].float().numpy(), n.numpy())
    for lay, state, t in zip(lays, (cache.key_cache_sp[0], cache.value_cache_sp[0]), types):
        assert state[0].dtype == t and state[4] == 212 and np.array_equal(state[3].cpu().numpy(), lay.ptr)
        assert np.array_equal(state[1][:, :212].cpu().numpy(), lay.lens)
        for r in range(B):
            assert np.array_equal(state[0][r, : lay.ptr[r]].float().cpu().numpy(), lay.flat[r])
    assert _common.read_status(torch.device("cuda")) == 0


def test_values_narrower_than_the_arenas_are_refused():
    x = torch.randn(1, 4, 256, dtype=torch.float32, device="cuda")
    lens = torch.full((1, 2, 4), 8, dtype=torch.int32, device="cuda")
    cache = CustomDynamicCache(arenas_per_batch=2, len_multiple=8)
    with pytest.raises(ValueError):
        cache.update_sp(x, lens, x[:, :, :128].contiguous(), lens, 256, 0, 128)
    assert cache.get_seq_length(0) == 0


@pytest.mark.parametrize("fresh", [False, True])
def test_a_block_whose_growth_fails_leaves_the_layer_as_it_was(fresh, monkeypatch):
    # K fits, the V buffer cannot grow (or be made): the block can be given again
    gen = torch.Generator().manual_seed(4)
    B, A, R = 2, 2, 128
    cache = CustomDynamicCache(arenas_per_batch=A, len_multiple=8)
    lays = [O.LayoutOracle(B * A, np.float32) for _ in range(2)]
    if not fresh:
        cache.reserve(0, B, 4000, 64, torch.bfloat16, "cuda")
    allocate = CustomDynamicCache._new_state if fresh else CustomDynamicCache._ensure_capacity
    for n_new, fails in ((20, fresh), (25, not fresh)):
        rows = [torch.randn(B, n_new, A * R, generator=gen).to(torch.bfloat16) for _ in range(2)]
        lens = [torch.full((B, A, n_new), n, dtype=torch.int32) for n in (16, 128)]
        args = (rows[0].cuda(), lens[0].cuda(), rows[1].cuda(), lens[1].cuda(), A * R, 0, R)
        if fails:
            calls = []

            def failing(*a):
                calls.append(a)
                if (len(calls) == 2 if fresh else a[0] is cache.value_cache_sp[0]):
                    raise torch.cuda.OutOfMemoryError("no memory")
                return allocate(*a)
            with monkeypatch.context() as m:
                m.setattr(cache, "_new_state" if fresh else "_ensure_capacity", failing)
                with pytest.raises(torch.cuda.OutOfMemoryError):
                    cache.update_sp(*args)
            for lst, lay in zip((cache.key_cache_sp, cache.value_cache_sp), lays):
                assert lst[0] is None if fresh else (lst[0][4] == 20 and np.array_equal(lst[0][3].cpu().numpy(), lay.ptr))
        cache.update_sp(*args)
        for lay, x, n in zip(lays, rows, lens):
            lay.update(x.float().view(B, n_new, A, R).permute(0, 2, 1, 3).reshape(B * A, n_new, R).numpy(), n.view(B * A, n_new).numpy())
    for lay, state in zip(lays, (cache.key_cache_sp[0], cache.value_cache_sp[0])):
        assert state[4] == 45 and np.array_equal(state[3].cpu().numpy(), lay.ptr)
        assert np.array_equal(state[1][:, :45].cpu().numpy(), lay.lens) and np.array_equal(state[2][:, :45].cpu().numpy(), lay.offs)
        for r in range(B * A):
            assert np.array_equal(state[0][r, : lay.ptr[r]].float().cpu().numpy(), lay.flat[r])
    assert _common.read_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("grows", ["both", "values"])
def test_ragged_blocks_grow_like_the_layout_oracle(grows):
    # rows of other counts in every block: at a growth some rows fit the old buffers (and moved on in the first attempt), some do not
    gen = torch.Generator().manual_seed(6)
    B, A, R = 3, 2, 128
    cache = CustomDynamicCache(arenas_per_batch=A, len_multiple=8)
    cache.reserve(0, B, 1 << 17 if grows == "values" else 1500, 8, torch.bfloat16, "cuda")
    if grows == "values":
        cache.value_cache_sp[0] = cache._new_state(B * A, 1500, 8, torch.bfloat16, "cuda")
    lays = [[O.LayoutOracle(A, np.float32) for _ in range(B)] for _ in range(2)]
    caps = []
    for n_new, counts in ((12, [12, 3, 0]), (70, [2, 70, 9]), (1, [1, 0, 1]), (300, [300, 1, 0]), (40, [40, 40, 40]), (5000, [17, 5000, 4097])):
        rows = [torch.randn(B, n_new, A * R, generator=gen).to(torch.bfloat16) for _ in range(2)]
        lens = [(torch.randint(0, 17, (B, A, n_new), generator=gen) * 8).to(torch.int32) for _ in range(2)]
        cache.update_sp(rows[0].cuda(), lens[0].cuda(), rows[1].cuda(), lens[1].cuda(), A * R, 0, R, token_counts=counts)
        for side in range(2):
            for b, c in enumerate(counts):
                lays[side][b].update(rows[side][b, :c].float().view(c, A, R).permute(1, 0, 2).numpy(), lens[side][b, :, :c].numpy())
        caps.append((cache.key_cache_sp[0][0].shape[1], cache.value_cache_sp[0][0].shape[1]))
    growths = [(a[0] != b[0], a[1] != b[1]) for a, b in zip(caps, caps[1:])]
    assert ((True, True) if grows == "both" else (False, True)) in growths
    stored = [lays[0][b].seq for b in range(B)]
    assert cache.seq_lens(0).tolist() == stored == cache.seq_lens_host(0)
    for side, state in enumerate((cache.key_cache_sp[0], cache.value_cache_sp[0])):
        assert state[5] == state[3].tolist() == [int(x) for b in range(B) for x in lays[side][b].ptr]
        for b in range(B):
            lay, n = lays[side][b], stored[b]
            assert np.array_equal(state[1][b * A:(b + 1) * A, :n].cpu().numpy(), lay.lens)
            assert np.array_equal(state[2][b * A:(b + 1) * A, :n].cpu().numpy(), lay.offs)
            for j in range(A):
                assert np.array_equal(state[0][b * A + j, : lay.ptr[j]].float().cpu().numpy(), lay.flat[j])
    assert _common.read_status(torch.device("cuda")) == 0
