"""CPU-only checks of the host side: router behaviour, C-ABI exports, loud failure without CUDA."""
import ctypes
import os
import re

import pytest
import torch

from dynakv_b200 import _lib
from dynakv_b200.kernels.router import KernelPolicy, compressed_decode_attention

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_default_kernel_boundary():
    policy = KernelPolicy()
    assert policy.select(0) == "short_fused"
    assert policy.select(499) == "short_fused"
    assert policy.select(500) == "long_two_stage"


def test_custom_kernel_boundary():
    policy = KernelPolicy(switch_tokens=128)
    assert policy.select(127) == "short_fused"
    assert policy.select(128) == "long_two_stage"


def test_negative_cache_length_is_rejected():
    with pytest.raises(ValueError):
        KernelPolicy().select(-1)


def test_policy_is_frozen_and_partitions_rows():
    policy = KernelPolicy()
    with pytest.raises(Exception):
        policy.switch_tokens = 3
    short, long_ = policy.partition([10, 499, 500, 32768, 0])
    assert short == [0, 1, 4] and long_ == [2, 3]


def test_library_exports_every_declared_symbol():
    header = open(os.path.join(ROOT, "include", "dynakv_b200.h")).read()
    declared = set(re.findall(r"^(?:int|size_t|const char\*)\s+(dkv_\w+)\s*\(", header, flags=re.M))
    assert declared, "no declarations found in the header"
    lib = _lib.load()
    for name in declared:
        assert hasattr(lib, name), f"{name} declared in include/dynakv_b200.h but not exported"
    assert declared == set(_lib.EXPORTS)
    assert lib.dkv_version() == 2


def test_struct_sizes_match_the_c_layout():
    # plain C layout: natural alignment, no packing
    assert ctypes.sizeof(_lib.Side) == 72
    assert ctypes.sizeof(_lib.AttnArgs) % 8 == 0
    assert _lib.AttnArgs.k.offset % 8 == 0 and _lib.AttnArgs.stream.offset % 8 == 0


def test_host_argument_errors_need_no_gpu():
    lib = _lib.load()
    a = _lib.AttnArgs()
    a.dtype, a.head_dim = 2, 64
    assert lib.dkv_fused_decode(ctypes.byref(a)) == -1
    assert b"head_dim" in lib.dkv_last_error()
    assert lib.dkv_fused_decode(None) == -1
    assert lib.dkv_split_workspace_bytes(None) == 0


def test_operators_refuse_cpu_tensors():
    q = torch.zeros(1, 4, 128)
    flat = torch.zeros(1, 8)
    lens = torch.zeros(1, 1, dtype=torch.int32)
    up = torch.zeros(4, 8, 128)
    with pytest.raises(RuntimeError, match="no CPU path"):
        compressed_decode_attention(q=q, k_flat=flat, k_up=up, v_flat=flat, v_up=up, key_lengths=lens,
                                    key_offsets=lens, value_lengths=lens, value_offsets=lens, theta=1e4,
                                    cache_length=1)


def test_two_stage_wrappers_require_offsets():
    from dynakv_b200.kernels.two_stage import abx_sparse, avx
    with pytest.raises(ValueError):
        abx_sparse(torch.zeros(1, 4, 128), torch.zeros(4, 8, 128), torch.zeros(1, 8), torch.zeros(1, 1, dtype=torch.int32))
    with pytest.raises(ValueError):
        avx(torch.zeros(1, 4, 1), torch.zeros(1, 8), torch.zeros(4, 8, 128), torch.zeros(1, 1, dtype=torch.int32))


def test_merge_basis_layout_matches_the_reference_rule():
    # reference: B[h, r, dd] = up[h*head_dim + dd, r] (kernels/compressed_attention.py:278-286, before the
    # repeat_interleave over query heads, which the kernels replace by head sharing)
    import torch
    from dynakv_b200.kernels.compressed_attention import merge_basis
    n_kv, d, rank = 3, 4, 12
    up = torch.arange(n_kv * d * rank, dtype=torch.float32).reshape(n_kv * d, rank)
    b = merge_basis(up, n_kv, d)
    assert b.shape == (n_kv, rank, d) and b.is_contiguous()
    for h in range(n_kv):
        for r in range(rank):
            for dd in range(d):
                assert b[h, r, dd] == up[h * d + dd, r]
    # the reference builds the same tensor as view -> transpose -> (repeat_interleave): compare with that recipe
    ref = up.view(n_kv, d, rank).transpose(1, 2)
    assert torch.equal(b, ref)
    low = merge_basis(up, n_kv, d, low_rank=5)
    assert torch.equal(low, ref[:, :5])


def test_balanced_sequence_partition_covers_every_sequence_and_balances_tokens():
    from dynakv_b200 import sharding, synthetic
    lengths = synthetic.log_uniform_lengths(64, 128, 32768, seed=3017)
    for world in (1, 2, 4, 8):
        parts = sharding.balanced_sequence_partition(lengths, world)
        assert sorted(i for p in parts for i in p) == list(range(64))
        loads = [sum(lengths[i] for i in p) for p in parts]
        assert max(loads) - min(loads) <= max(lengths)          # longest-first greedy bound
        assert max(loads) <= 1.25 * sum(lengths) / world or world == 1 or max(lengths) > sum(lengths) / world
    assert sharding.balanced_sequence_partition([5, 5], 4) == [[0], [1], [], []]


def test_ctypes_mirrors_have_the_c_compilers_layout(tmp_path):
    """Every struct of include/dynakv_b200.h, field by field: size and offsets as gcc lays them out against the
    ctypes mirror in dynakv_b200/_lib.py (same field names, same order)."""
    import os
    import shutil
    import subprocess
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no C compiler")
    pairs = {"dkv_side": _lib.Side, "dkv_attn_args": _lib.AttnArgs, "dkv_append_args": _lib.AppendArgs,
             "dkv_pack_args": _lib.PackArgs, "dkv_project_args": _lib.ProjectArgs, "dkv_gate_args": _lib.GateArgs}
    lines = ["#include <stdio.h>", "#include <stddef.h>", '#include "dynakv_b200.h"', "int main(void) {"]
    for cname, cls in pairs.items():
        lines.append(f'  printf("{cname} size %zu\\n", sizeof({cname}));')
        for fname, _ in cls._fields_:
            lines.append(f'  printf("{cname} {fname} %zu\\n", offsetof({cname}, {fname}));')
    lines += ["  return 0;", "}"]
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines))
    exe = tmp_path / "layout"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")
    subprocess.run([gcc, "-std=c99", "-I", inc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    seen = 0
    for line in out.splitlines():
        cname, what, value = line.split()
        cls = pairs[cname]
        if what == "size":
            assert ctypes.sizeof(cls) == int(value), (cname, ctypes.sizeof(cls), value)
        else:
            assert getattr(cls, what).offset == int(value), (cname, what)
        seen += 1
    assert seen == sum(len(c._fields_) + 1 for c in pairs.values())


def test_waits_of_the_decode_pipeline_answer_for_a_whole_warp():
    """Shuffles, votes, tensor-memory accesses and elected lanes follow the waits: no lane may leave one, or go on, by itself."""
    source = open(os.path.join(ROOT, "dynakv_b200", "csrc", "dkv_mma_decode.cu")).read()
    waits = dict(re.findall(r"__device__ __forceinline__ bool (mbar_wait\w*)\([^)]*\) \{\n(.*?)\n\}", source, flags=re.S))
    assert waits
    for name, body in waits.items():
        exits = re.findall(r"[^\n]*\breturn (?:true|ok)\b[^\n]*|if \([^\n]*abort_flag[^\n]*", body)
        assert len(exits) >= 2 and all("_sync(0xffffffffu" in e for e in exits), name
    # and nothing else polls a barrier
    assert source.count("mbar_test(") == 1 + len(waits)


def test_a_decode_kernel_that_gives_up_waits_for_what_is_in_flight():
    """Copies and products end before shared memory and tensor memory go, also when the loops were left by waits that ran out."""
    source = open(os.path.join(ROOT, "dynakv_b200", "csrc", "dkv_mma_decode.cu")).read()
    body = re.search(r"void end_what_is_in_flight\([^)]*\) \{(.*?)\n\}\n", source, flags=re.S).group(1)
    order = [body.index(w) for w in ("cp_async_wait_all()", "umma_commit(", "mbar_wait(", "__syncthreads()")]
    assert order == sorted(order)
    end = source[source.index("// ---- epilogue"):source.index("tcgen05.dealloc")]
    assert re.search(r"__syncthreads\(\);\n  if \(\*abort_flag\) end_what_is_in_flight\(", end)


def test_kernels_that_overlap_the_append_read_its_cache_with_ordinary_loads():
    """A read-only load is for data that nothing writes in the kernel's lifetime: here the V basis alone."""
    for name in ("dkv_mma_decode.cu", "dkv_short.cu"):
        source = open(os.path.join(ROOT, "dynakv_b200", "csrc", name)).read()
        loads = re.findall(r"[^\n]*(?:__ldg\(|ld\.global\.nc)[^\n]*", source)
        assert all("vup" in line for line in loads), loads


@pytest.mark.parametrize("switch,longest", [(1, 0), (2, 256), (64, 256), (129, 256), (130, 512), (300, 768), (385, 768), (386, 1024), (500, 1024),
                                            (2000, 1024), (2 ** 31 - 1, 1024)])
def test_switch_point_decides_in_a_routed_call(switch, longest):
    """One kernel for rows of any length only up to twice the tiles of the longest row that the policy calls short."""
    a = _lib.AttnArgs()
    a.dtype, a.batch, a.n_q_heads, a.n_basis_groups, a.arenas_per_batch, a.head_dim, a.rank, a.len_multiple = _lib.DKV_BF16, 4, 32, 8, 8, 128, 128, 8
    for side in (a.k, a.v):
        side.flat_stride, side.lens_stride_s, side.offs_stride_s = 8, 1, 1
    a.n_sm = 148
    for columns in (1, 128, 129, 256, 257, 499, 512, 513, 768, 769, 1000, 1024, 1025, 4096):
        a.seq_len = columns
        n = _lib.load().dkv_routed_launches(ctypes.byref(a), switch)
        assert (n == 1) == (columns <= longest), (columns, n)


def test_quotient_from_a_reciprocal_and_two_remainders_is_the_division():
    """The gate's division of exponentials by their row's sum, step by step in exact arithmetic."""
    from fractions import Fraction

    import numpy as np

    def rn(f):          # to the nearest float32, ties to even
        if f == 0:
            return Fraction(0)
        n, e = abs(f), 0
        while n >= 2 ** 24:
            n, e = n / 2, e + 1
        while n < 2 ** 23 and e > -149:
            n, e = n * 2, e - 1
        return (1 if f > 0 else -1) * Fraction(round(n)) * Fraction(2) ** e

    def quotient(a, b):
        y = rn(1 / b)
        q = rn(a * y)
        for _ in range(2):
            q = rn(rn(a - q * b) * y + q)
        return q

    rng = np.random.default_rng(5)
    for lowest, exact in ((-100, True), (-148, False)):
        for _ in range(1500):
            a = rn(Fraction(float(rng.uniform(1, 2))) * Fraction(2) ** int(rng.integers(lowest, 0)))
            b = rn(Fraction(float(rng.uniform(1, 1024))))
            want, got = rn(a / b), quotient(a, b)
            assert got == want if exact else abs(got - want) <= max(want / 2 ** 23, Fraction(2) ** -149)


def test_smoke_check_reaches_the_split_kernel():
    import __graft_entry__ as entry
    a = _lib.AttnArgs()
    a.dtype, a.batch, a.n_q_heads, a.n_basis_groups, a.arenas_per_batch, a.head_dim, a.rank, a.len_multiple = _lib.DKV_BF16, 2, 32, 8, 8, 128, 128, 8
    for side in (a.k, a.v):
        side.flat_stride, side.lens_stride_s, side.offs_stride_s = 8, 1, 1
    a.n_sm, a.seq_len = 148, max(entry.SMOKE_TOKENS) + 8
    switch = KernelPolicy().switch_tokens
    assert len(entry.SMOKE_TOKENS) == 2 and min(entry.SMOKE_TOKENS) + 1 < switch <= max(entry.SMOKE_TOKENS)
    assert 1 + _lib.load().dkv_routed_launches(ctypes.byref(a), switch) == entry.SMOKE_LAUNCHES
