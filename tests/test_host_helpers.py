"""Host-side choices that need no GPU: how the decode attention's keys are split over CTAs, the uniform numbers of
sampling, the size limit of the L2 hints."""
from __future__ import annotations

import os
import random
import subprocess
import sys

import torch

from cuinfer_b200 import kernels
from cuinfer_b200.sampling.sampler import uniform


def test_decode_splits_is_sane_for_every_shape():
    rnd = random.Random(0)
    for _ in range(400):
        requests = rnd.choice([1, 2, 3, 5, 8, 12, 17, 32, 64, 200])
        kv_heads = rnd.choice([1, 2, 4, 8, 16])
        keys = rnd.choice([1, 15, 64, 65, 500, 1024, 4096, 5000, 32768, 131072])
        for tma in (False, True):                               # the cache layout allows the TMA path or not
            s = kernels.decode_splits(requests, kv_heads, keys, tma=tma)
            assert 1 <= s <= 64
            if s > 1:
                share = -(-(-(-keys // s)) // 64) * 64        # keys per CTA, in steps of 64
                assert (s - 1) * share < keys                   # the last CTA still has keys to read
    # few (request, kv head) pairs and many keys: split; the GPU already full of pairs: do not
    assert kernels.decode_splits(1, 8, 4096) > 8 and kernels.decode_splits(8, 8, 4096) >= 2
    assert kernels.decode_splits(64, 8, 4096) == 1 and kernels.decode_splits(256, 8, 512) == 1
    assert kernels.decode_splits(1, 8, 16) == 1                 # one block of keys cannot be shared
    # 24 requests x 8 heads leave a third of the GPU free, but a second round of CTAs would cost more than it brings
    assert kernels.decode_splits(24, 8, 2048, tma=True) == 1 and kernels.decode_uses_tma(2048, 1)
    assert not kernels.decode_uses_tma(4096, 32)                # short streams per CTA stay on cp.async
    # more keys never mean fewer CTAs for the same batch
    for requests in (1, 2, 8):
        counts = [kernels.decode_splits(requests, 8, n) for n in (256, 1024, 4096, 16384)]
        assert counts == sorted(counts)


def test_the_choice_of_splits_knows_which_launches_merge_in_clusters():
    """The host's estimate and the kernel's launch take the same launches for clusters, whatever the group and head size; the
    choice is the one that the merge really taken calls for."""
    lib = kernels.library()
    for pairs in (1, 2, 3, 8, 16, 18, 19, 24, 37, 49, 50, 74, 75, 148, 149, 500):
        for splits in (1, 2, 3, 4, 5, 6, 7, 8, 9, 16):
            for group in (1, 2, 3, 4, 6, 8, 16):
                for head_dim in (64, 128, 256):
                    for tma in (False, True):
                        assert kernels.decode_merges_in_cluster(pairs, splits, group, head_dim, tma) == bool(
                            lib.cib_decode_merges_in_cluster(pairs, splits, group, head_dim, int(tma))), (pairs, splits, group, head_dim, tma)
    # groups of two heads of 128 meet in clusters of eight; the partials of groups of four and more do not fit, and the merge
    # through memory that they then take asks for more and shorter shares
    assert kernels.decode_splits(2, 8, 2048, group=2) == 8 and kernels.decode_splits(2, 8, 2048, group=4) == 16
    assert kernels.decode_splits(1, 8, 512, group=4) == 4 and kernels.decode_splits(1, 8, 1500, group=4) == 24


def test_uniform_numbers_depend_on_seed_request_and_index_only():
    seen = set()
    for seed in (0, 1, 12345):
        for key in (0, 7, 2 ** 40 + 3):
            for index in range(50):
                u = uniform(seed, key, index)
                assert 0.0 <= u < 1.0 and u == uniform(seed, key, index)
                assert u * (1 << 24) == int(u * (1 << 24))      # 24 random bits: exact in float32
                seen.add(u)
    assert len(seen) > 440                                      # 450 draws, (almost) all different
    draws = [uniform(3, 9, i) for i in range(4000)]
    assert 0.47 < sum(draws) / len(draws) < 0.53
    assert 0.22 < sum(d < 0.25 for d in draws) / len(draws) < 0.28


def test_l2_hints_are_given_for_small_weights_only():
    small = torch.empty(1024, 1024, dtype=torch.bfloat16)
    large = torch.empty(kernels.L2_HINT_MAX_BYTES // 2 + 8, dtype=torch.bfloat16)
    assert kernels._l2_hint(small) is small and kernels._l2_hint(large) is None and kernels._l2_hint(None) is None


def test_step_buckets_hold_their_batches_with_little_to_spare():
    """The sizes a step is padded to before it runs as a captured graph: never smaller than the batch, one request to
    spare for the spare tokens, at most an eighth (or 15) more tokens, and few distinct buckets."""
    from cuinfer_b200.engine.runner import ModelRunner
    from cuinfer_b200.parts.context import StepContext

    rnd = random.Random(1)
    seen = set()
    for _ in range(3000):
        R = rnd.choice([1, 1, 2, 3, 8, 17, 33, 100, 255])
        lens = [rnd.choice([1, 1, 1, 2, 7, 60, 500, 2000]) for _ in range(R)]
        wants = [rnd.choice([0, 1, 1, 2]) for _ in range(R)]
        T, S = sum(lens), sum(wants)
        Tb, Rb, Sb = ModelRunner.step_bucket(lens, wants)
        assert T <= Tb <= max(T + 15, T + T // 8 + 1) and Tb % 16 == 0
        assert R < Rb <= 2 * R and Rb & (Rb - 1) == 0
        assert S <= Sb <= max(2 * S - 1, Rb if S else 0) and Sb & (Sb - 1) == 0
        seen.add(Tb)
        # what a recorded step's launches are sized by: at most so many row tiles, and at least so many, in every batch
        least_tokens, least_requests = ModelRunner.step_bucket_least(Tb, Rb)
        assert least_tokens <= T and least_requests <= R
        ctx = StepContext.__new__(StepContext)
        ctx.launch_query_lens, ctx.launch_least = [Tb + 128] + [1] * (Rb - 1), (least_tokens, least_requests)
        for g in (1, 2, 3, 4, 8, 16):
            tiles = sum(-(-n * g // 128) for n in lens)
            assert ctx.least_row_tiles(g, 128) <= tiles <= sum(-(-n * g // 128) for n in ctx.query_lens_for_launch())
    assert len(seen) < 120
    assert ModelRunner.step_bucket([2048], [1]) == (2048, 2, 2) and ModelRunner.step_bucket([8192], [1])[0] == 8192


def test_decode_products_that_share_nothing_leave_the_library_only_where_it_is_slower(monkeypatch):
    """17 to 32 rows whose product has neither a norm nor a gate beside it: streamed where the library has to split K, or for
    32-bit rows; everything else goes to the library, up to 16 rows nothing does."""
    from cuinfer_b200.parts import gemm_dispatch
    streamed = []
    monkeypatch.setattr(kernels, "gemm_wstream", lambda x, w, out: streamed.append(w.shape))
    for M, N, K, dtype, own in [(24, 192, 64, torch.bfloat16, True), (32, 256, 512, torch.bfloat16, True), (17, 512, 1024, torch.bfloat16, True),
                                (24, 512, 512, torch.bfloat16, False), (32, 1024, 256, torch.bfloat16, False), (17, 1024, 1024, torch.bfloat16, False),
                                (24, 264, 520, torch.bfloat16, False), (33, 512, 1024, torch.bfloat16, False), (24, 1024, 256, torch.float32, True),
                                (9, 128, 4104, torch.bfloat16, True)]:
        x, w = torch.ones(M, K, dtype=torch.bfloat16), torch.ones(N, K, dtype=torch.bfloat16)
        if dtype == torch.bfloat16 or own:                      # (the library's 32-bit store of bfloat16 rows is for CUDA tensors)
            out = torch.zeros(M, N, dtype=dtype)
            streamed.clear()
            gemm_dispatch.bf16_matmul_nt(x, w, out)
            assert streamed == ([w.shape] if own else []), (M, N, K)
            assert own or bool((out == K).all())
        assert gemm_dispatch.plain_takes_wstream(M, N, K, dtype) is own


def test_gated_decode_products_without_a_shared_norm_are_streamed_up_to_32_rows(monkeypatch):
    from cuinfer_b200.parts.base import LazyNorm, ResidualStream
    from cuinfer_b200.parts.linear import Linear

    class PlainNorm:
        def add_norm(self, stream):
            return stream.residual.to(torch.bfloat16)

    called = []
    monkeypatch.setattr(kernels, "gemm_wstream", lambda x, w, out, silu_pair=False, **kw: called.append(("streamed", bool(silu_pair))))
    monkeypatch.setattr(kernels, "silu_mul", lambda y, act, gelu=False: called.append(("gate", gelu)))
    product = Linear(["w"], [1024], 256, torch.bfloat16)
    product.weight = torch.ones(1024, 256, dtype=torch.bfloat16)
    for M, own in [(17, True), (32, True), (33, False), (64, False)]:
        for x in (torch.ones(M, 256, dtype=torch.bfloat16), LazyNorm(ResidualStream(torch.ones(M, 256)), PlainNorm())):
            called.clear()
            assert product.forward(x, silu_pair=True).shape == (M, 512)
            assert called == ([("streamed", True)] if own else [("gate", False)]), (M, type(x))


def test_row_tiles_without_the_requests_of_one_token():
    """What a recorded step says that it has at least when another kernel takes its single tokens."""
    from cuinfer_b200.engine.runner import ModelRunner
    from cuinfer_b200.parts import StepContext
    rnd = random.Random(4)
    for _ in range(3000):
        R = rnd.choice([1, 2, 3, 8, 17, 33, 100, 255])
        lens = [rnd.choice([1, 1, 1, 1, 2, 7, 60, 500]) for _ in range(R)]
        Tb, Rb, _ = ModelRunner.step_bucket(lens, [1] * R)
        ctx = StepContext.__new__(StepContext)
        ctx.num_requests = Rb
        ctx.launch_query_lens, ctx.launch_least = [Tb + 128] + [1] * (Rb - 1), ModelRunner.step_bucket_least(Tb, Rb)
        for g in (1, 2, 4, 16):
            assert ctx.least_row_tiles(g, 128, True) <= sum(-(-n * g // 128) for n in lens if n > 1), (lens, g)
    ctx.num_requests, ctx.launch_least = 32, (2017, 16)
    assert ctx.least_row_tiles(2, 128, True) == 32 and ctx.least_row_tiles(2, 128) == 32 and ctx.least_row_tiles(16, 128, True) == 249


def test_single_tokens_of_a_mixed_step_are_computed_apart_only_where_that_pays(monkeypatch):
    """Recorded steps that do not say that they hold many single tokens launch the prompt kernel alone; so do steps whose single
    tokens fit the SMs beside the portions, and long portions beside short contexts."""
    from cuinfer_b200.parts import GroupView, PagedKV, StepContext, attention_dispatch
    launched = []
    monkeypatch.setattr(kernels, "attention_tcgen05", lambda *a, least_tiles, least_query: launched.append(("prompt", least_tiles, least_query)))
    monkeypatch.setattr(kernels, "paged_attention_decode", lambda *a, query_start_loc=None, **kw: launched.append(("single", query_start_loc is not None)))
    assert attention_dispatch.singles_apart_from(torch.bfloat16, 16, 8, 128) == 19
    assert attention_dispatch.singles_apart_from(torch.float32, 16, 8, 128) is None

    def kinds(lens, keys=300, recorded=None, window=0):
        starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
        i32 = lambda x: torch.tensor(x, dtype=torch.int32)
        held = [keys if n == 1 else n for n in lens]
        ctx = StepContext(starts[-1], len(lens), None, None, None, i32(starts), i32(held), None, query_start_loc_host=starts, seq_lens_host=held,
                          max_seq_len=max(held))
        if recorded is not None:
            ctx.query_start_loc_host = ctx.seq_lens_host = None
            ctx.num_requests, ctx.launch_singles, ctx.launch_least = 32, recorded, (max(1, sum(lens) - 15), 16)
            ctx.launch_query_lens = [sum(lens) + 128] + [1] * 31
        rows = torch.empty(starts[-1], 32 * 128, dtype=torch.bfloat16)
        kv = PagedKV(torch.empty(2, 2, 8, 16, 128, dtype=torch.bfloat16), GroupView(16, i32([[0]] * len(lens)), None))
        launched.clear()
        attention_dispatch.paged_attention(rows, torch.empty(starts[-1], 16 * 128, dtype=torch.bfloat16), kv, ctx, 16, 8, 128, 0.1, window)
        assert launched[-1][0] == "prompt" and launched[-1][2] == len(launched)
        return len(launched)

    assert kinds([60] * 24, recorded=0) == 1 and kinds([1] * 18 + [60] * 3, recorded=0) == 1       # (recorded for fewer than 19)
    assert kinds([1] * 19 + [60] * 3, recorded=19) == 2 and launched == [("single", True), ("prompt", 3, 2)]
    assert kinds([60] * 24) == 1 and kinds([1] * 18 + [60] * 3) == 1 and kinds([1] * 19 + [60] * 3) == 2
    # more than three row tiles an SM: by the contexts, where they are known
    assert kinds([1] * 23 + [3400]) == 2 and kinds([1] * 23 + [5000]) == 1 and kinds([1] * 23 + [5000], keys=2048) == 2
    assert kinds([1] * 23 + [5000], keys=4000, window=1024) == 1 and kinds([1] * 23 + [3900], recorded=19) == 1


def test_no_product_runs_as_pairs_of_ctas_when_they_are_switched_off():
    code = "from cuinfer_b200 import kernels; print(kernels.gemm_tcgen05_stream_cols(8192, 1024, 1024))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    cols = [subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, CUINFER_B200_GEMM_PAIR=on), capture_output=True, text=True,
                           timeout=600, check=True).stdout.split() for on in ("1", "0")]
    assert cols == [["256"], ["0"]]


def test_a_product_with_a_bias_takes_a_norm_that_has_not_been_computed(monkeypatch):
    """As every projection does: the rows are normed first."""
    from cuinfer_b200.parts.base import LazyNorm, ResidualStream
    from cuinfer_b200.parts.linear import Linear
    added = []
    monkeypatch.setattr(Linear, "forward", lambda self, x: torch.zeros(x.shape[0], 8192, dtype=torch.bfloat16))
    monkeypatch.setattr(kernels, "bias_rows", lambda y, bias, out, squared_relu=False: added.append((tuple(y.shape), squared_relu)))
    product = Linear(["w"], [8192], 4096, torch.bfloat16)
    product.weight = torch.zeros(8192, 4096, dtype=torch.bfloat16)
    product.forward_biased(LazyNorm(ResidualStream(torch.zeros(3, 4096)), None), torch.zeros(8192), squared_relu=True)
    assert added == [((3, 8192), True)]
