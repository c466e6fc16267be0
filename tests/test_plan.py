"""The product planner (host code of the tensor-core library, callable without a GPU): whatever it chooses for a
step of up to `chunk` tokens fits the scratch an engine reserves for that chunk size from sizes alone, at the
benchmark's layer shapes, a small model's and odd ones; and a few of the choices that the measurements in
`profiles/` rest on."""
import pytest

from mdma_b200 import ops_tensor

STORE, ACCUMULATE, GATED = 0, 1, 2
SHAPES = {          # name -> [(mode, features, K)]
    "8b": [(STORE, 6144, 4096), (ACCUMULATE, 4096, 4096), (GATED, 14336, 4096), (ACCUMULATE, 4096, 14336), (STORE, 128256, 4096)],
    "7b": [(STORE, 12288, 4096), (ACCUMULATE, 4096, 4096), (GATED, 11008, 4096), (ACCUMULATE, 4096, 11008), (STORE, 32000, 4096)],
    "1b": [(STORE, 3072, 2048), (ACCUMULATE, 2048, 2048), (GATED, 8192, 2048), (ACCUMULATE, 2048, 8192), (STORE, 128256, 2048)],
    "odd": [(STORE, 520, 264), (ACCUMULATE, 136, 2048), (GATED, 331, 640), (ACCUMULATE, 5000, 72), (STORE, 97, 8)],
}


@pytest.mark.parametrize("sms", [148, 132, 78])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_every_plan_fits_the_scratch_reserved_for_its_chunk_size(name, sms):
    tokens = list(range(1, 300)) + list(range(300, 1200, 7)) + [2048, 4096, 8191, 8192]
    for m in tokens:
        bound = ops_tensor.scratch_floats_bound(sms, m, 1, ())
        for mode, n, k in SHAPES[name]:
            bn, splits = ops_tensor.gemm_plan(mode, m, n, k, sms)
            assert bn in (16, 32, 64, 128, 256, 512) and (splits >= 1 or splits in (-2, -3, -4)), (m, mode, n, k, bn, splits)
            if bn != 512:
                assert bn >= min(m, 256) or m > 128, (m, bn)          # a token tile covers the step, or the step is tiled
            need = ops_tensor.gemm_scratch_floats(bn, splits, m, n, sms)
            assert need <= bound, f"{name}: {m} tokens, mode {mode}, {n} x {k}: plan ({bn}, {splits}) needs {need} floats, {bound} reserved"


def test_choices_that_the_measurements_rest_on():
    plan = lambda mode, m, n, k: ops_tensor.gemm_plan(mode, m, n, k, 148)
    assert plan(STORE, 8, 6144, 4096) == (16, 4)             # QKV at batch 8: four splits (the next kernel adds them up itself)
    assert plan(ACCUMULATE, 8, 4096, 4096) == (16, 9)        # O: two blocks per SM
    assert plan(GATED, 8, 14336, 4096) == (16, -2)           # gate+up: K split inside a cluster of two
    assert plan(GATED, 64, 14336, 4096) == (64, 1)
    assert [plan(GATED, m, 5632, 2048) for m in (33, 48, 64)] == [(64, 1)] * 3        # in a decode step pairs, which do not start early, lose
    assert plan(GATED, 128, 14336, 4096)[0] == 512           # block pairs from 97 tokens
    assert plan(ACCUMULATE, 256, 4096, 14336) == (256, 4)    # down of 256 tokens: one wide token tile, four splits
    assert plan(STORE, 256, 6144, 4096) == (128, 1)          # QKV stays unsplit there (its partial sums cost the rotary kernel more)
    assert plan(GATED, 2048, 14336, 4096) == (512, 1) and plan(STORE, 2048, 6144, 4096) == (512, 1)
    assert plan(STORE, 8, 128256, 4096) == (16, 1)           # the head: more tiles than SMs, no split


def test_block_pairs_divide_k_only_where_a_norm_adds_the_parts_up():
    plan = lambda m, n, k, folded: ops_tensor.gemm_plan(ACCUMULATE, m, n, k, 148, folded)  # noqa: E731
    for m, n, k, splits in ((513, 2048, 2048, 3), (768, 2048, 8192, 3), (1024, 2048, 8192, 2), (768, 1024, 4096, 6), (2048, 1024, 4096, 2), (600, 1000, 1024, 4),
                            (512, 4096, 4096, 2), (385, 4096, 4096, 2), (384, 4096, 14336, 2), (257, 4096, 14336, 2)):
        assert plan(m, n, k, True) == (512, splits), (m, n, k)
        bn, alone = plan(m, n, k, False)
        assert (bn, alone) == (512, 1) if m > 512 else bn != 512, (m, n, k)
    # ... nor of 257-512 tokens where the one-block kernel is faster, up to 256 tokens, or without idle pairs; never a stored product
    for m, n, k in ((512, 2048, 2048), (384, 4096, 4096), (384, 2048, 2048), (256, 4096, 14336), (1500, 2048, 2048)):
        assert plan(m, n, k, True) == plan(m, n, k, False) and (plan(m, n, k, True)[0] != 512 or plan(m, n, k, True)[1] == 1)
    assert ops_tensor.gemm_plan(STORE, 768, 3072, 2048, 148) == (512, 1)
    for m in range(257, 2049, 13):
        for mode, n, k in SHAPES["1b"] + SHAPES["odd"]:
            if mode == ACCUMULATE:
                bn, splits = plan(m, n, k, True)
                assert ops_tensor.gemm_scratch_floats(bn, splits, m, n, 148) <= ops_tensor.scratch_floats_bound(148, m, 1, ())


def test_a_stored_product_in_front_of_a_norm_takes_wide_token_tiles():
    """... as an added one does; the products that the rotary write reads stay as they were."""
    plan = lambda m, n, k, folded: ops_tensor.gemm_plan(STORE, m, n, k, 148, folded)  # noqa: E731
    for m, n, k, want in ((160, 4096, 16384, (256, 4)), (256, 4096, 16384, (256, 4)), (512, 4096, 16384, (256, 2)), (130, 2048, 8192, (256, 9)),
                          (400, 2048, 8192, (256, 4)), (300, 4096, 4096, (256, 2)), (160, 1536, 6144, (128, 6)), (160, 2048, 2048, (128, 4))):
        assert plan(m, n, k, True) == want and plan(m, n, k, False)[0] == 128, (m, n, k)
        assert ops_tensor.gemm_scratch_floats(*want, m, n, 148) <= ops_tensor.scratch_floats_bound(148, m, 1, ())
    assert plan(256, 6144, 4096, False) == (128, 1)


def test_a_sublayer_says_whether_its_sums_are_added_up():
    """Nested arrangements: one that does not add up holds for all that it contains, and the state is as before after an error."""
    from types import SimpleNamespace
    import torch
    from mdma_b200.parts.base import Runtime
    tc = SimpleNamespace(folds=True)
    rt = Runtime(torch.bfloat16, torch.device("cpu"), "tensor", tc=tc)
    seen = lambda: tc.folds  # noqa: E731
    assert rt.unfolded(rt.unfolded, seen) is False and tc.folds is True
    assert rt.unfolded(lambda: (rt.unfolded(seen), seen())) == (False, False) and tc.folds is True
    with pytest.raises(KeyError):
        rt.unfolded({}.__getitem__, 0)
    assert tc.folds is True
    assert Runtime(torch.float32, torch.device("cpu")).unfolded(lambda: 5) == 5


def test_clusters_that_start_early_have_two_blocks():
    """A cluster is placed as ordinary blocks are up to two blocks; wider ones are launched in stream order and never planned."""
    from mdma_b200.csrc import build
    early = build.load("tensor").mdma_gemm_tc_starts_early
    assert [early(c) for c in (3, 4, 8)] == [0, 0, 0]
    for m in (1, 8, 16, 17, 32):
        for n, k in ((8192, 2048), (5632, 2048), (2752, 1024), (8192, 3072), (331, 640), (14336, 4096), (128, 65536)):
            assert ops_tensor.gemm_plan(GATED, m, n, k, 148)[1] in (-2, 1), (m, n, k)


@pytest.mark.parametrize("sms", [148, 78])
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 128), (32, 32, 128), (32, 8, 64), (16, 8, 16), (6, 3, 48), (64, 1, 32), (40, 2, 64)])
def test_every_choice_of_key_splits_fits_the_scratch_reserved_for_attention(heads, kv_heads, head_dim, sms):
    """The attention kernels keep tokens x heads x splits x (head_dim + 2) floats when they split the keys; the
    engine reserves a bound computed from sizes alone.  Every (sequences, tokens per sequence, context, capacity)
    the step function can see must stay below it."""
    reserved = (ops_tensor.scratch_floats_bound(sms, 8192, 1, [(heads, kv_heads, head_dim)])
                - ops_tensor.scratch_floats_bound(sms, 8192, 1, ()))
    worst = 0
    for n_seqs in list(range(1, 40)) + [48, 64, 100, 148, 200, 300, 600]:
        for max_new in (1, 2, 5, 16, 17, 64, 129, 700):
            if n_seqs * max_new > 8192:
                continue
            for max_len in (1, 64, 580, 1024, 1025, 4096, 40000):
                if max_len < max_new:
                    continue
                for most in (None, n_seqs, max(n_seqs, 64)):
                    splits = ops_tensor.attention_splits(n_seqs, max_new, max_len, heads, kv_heads, sms, most)
                    assert 1 <= splits <= 32
                    need = n_seqs * max_new * heads * splits * (head_dim + 2) if splits > 1 else 0
                    worst = max(worst, need)
                    assert need <= reserved, (n_seqs, max_new, max_len, most, splits, need, reserved)
    assert worst > 0          # the sweep did reach split cases


def test_contexts_of_one_tile_a_warp_are_not_divided():
    """An engine for a handful of sequences whose longest context is one tile for each of a block's twelve warps: no pieces,
    whatever its sequences hold; a longer one is cut as before."""
    splits = lambda most_len, dim: {ops_tensor.attention_splits(n, 1, length, 32, 8, 148, 2, most_len, dim) for n in (1, 2) for length in (1, 64, most_len)}  # noqa: E731
    assert splits(384, 128) == {1} and splits(768, 64) == {1} and splits(100, 64) == {1}
    assert splits(385, 128) == {4} and splits(769, 64) == {4} and splits(1000, 128) == {4}
    assert ops_tensor.attention_splits(1, 1, 100, 32, 8, 148, 2) == 4

def test_short_rows_of_one_matrix_are_not_streamed():
    """A block's stages are as long as a chunk of runs: one matrix streams where K fills it, or where there is enough of W."""
    from mdma_b200.csrc import build
    streams = lambda n, k, gated=0: build.load("core").mdma_gemm_simt_streams(n, k, gated, 148)  # noqa: E731
    for n, k in ((9472, 64), (9472, 128), (9472, 384), (14000, 384), (20000, 256), (32000, 64), (32000, 128), (4736, 520), (4736, 768), (7000, 640)):
        assert streams(n, k) == 0, (n, k)
    for n, k in ((32000, 1024), (32000, 512), (32000, 256), (20000, 384), (128256, 64), (4736, 1024), (4739, 1000), (9472, 512), (128256, 768)):
        assert streams(n, k) == 1, (n, k)
    assert streams(9472, 64, 1) == streams(4736, 520, 1) == streams(2368, 1024, 1) == 1
    assert [streams(*c) for c in ((4728, 1024), (9456, 512), (2364, 1024, 1), (200000, 1028), (200000, 1022))] == [0] * 5
