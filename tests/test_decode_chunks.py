"""Single-token steps whose sequences' keys are cut into pieces of one size (`decode_chunks`)."""
import math

import pytest
import torch


@pytest.mark.parametrize("sms", [148, 78])
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 128), (32, 32, 128), (16, 8, 16), (64, 64, 64), (40, 2, 64)])
def test_pieces_cover_the_context_and_fit_the_scratch(heads, kv_heads, head_dim, sms):
    from mdma_b200 import ops_tensor
    reserved = (ops_tensor.scratch_floats_bound(sms, 8192, 1, [(heads, kv_heads, head_dim)])
                - ops_tensor.scratch_floats_bound(sms, 8192, 1, ()))
    seen = 0
    for n_seqs in range(1, 200):
        for max_len in (1, 1024, 1025, 2048, 3000, 9000, 40000):
            splits, keys = ops_tensor.decode_chunks(n_seqs, max_len, kv_heads, sms)
            if splits == 1:
                assert keys == 0
                continue
            seen += 1
            assert keys % 64 == 0 and splits * keys >= max_len and n_seqs * kv_heads >= sms
            assert n_seqs * heads * splits * (head_dim + 2) <= reserved
    assert seen


@pytest.mark.parametrize("most_seqs,most_len,kv_heads", [(8, 8192, 32), (8, 2041, 32), (24, 4096, 8), (37, 131072, 4), (5, 40000, 32)])
def test_a_piece_is_as_long_whoever_the_batch_mates_are(most_seqs, most_len, kv_heads):
    """From the engine's capacity: a live batch that shrinks, or whose longest sequence grows, changes the number of pieces only;
    full engines at their whole context fit the scratch."""
    from mdma_b200 import ops_tensor
    sms, lengths = 148, set()
    for n_seqs in range(1, most_seqs + 1):
        for max_len in range(1024, -(-most_len // 1024) * 1024 + 1, 1024):
            splits, keys = ops_tensor.decode_chunks(n_seqs, max_len, kv_heads, sms, most_seqs, most_len)
            assert n_seqs * kv_heads * splits <= 5 * sms or splits == 1
            if splits > 1:
                lengths.add(keys)
                assert n_seqs * kv_heads >= sms and (splits - 1) * keys < max_len <= splits * keys
                # where one piece holds them all, nothing is cut: the same arithmetic without the merge
                assert ops_tensor.decode_chunks(n_seqs, keys, kv_heads, sms, most_seqs, most_len) == (1, 0)
    assert len(lengths) == 1 and next(iter(lengths)) % 1024 == 0


@pytest.mark.gpu
@pytest.mark.parametrize("H,K,hd", [(4, 4, 128), (8, 2, 64), (6, 6, 48)])
@pytest.mark.parametrize("splits,keys", [(2, 64), (5, 128), (16, 64), (2, 1024)])
def test_decode_in_pieces(H, K, hd, splits, keys):
    """Against float64 at lengths around the pieces' edges; a piece that a sequence does not reach leaves nothing behind."""
    from mdma_b200 import ops_tensor
    from mdma_b200.parts.rotary import inverse_frequencies
    from test_kernels import DEV, StepMeta, close, fill_cache, ops_mod, reference_attention
    ops = ops_mod()
    torch.manual_seed(H + hd + keys)
    page, most = 64, splits * keys
    cached = [min(c, most - 1) for c in (0, keys - 2, keys - 1, keys, 2 * keys - 1, most - 1, 31)]
    B = len(cached)
    lens = [c + 1 for c in cached]
    kc, vc, table, max_pages, dense = fill_cache(lens, K, hd, page, torch.bfloat16, seed=hd, poison=True)
    inv_freq = inverse_frequencies(hd, 10000.0).to(DEV)
    qkv = torch.randn(B, (H + 2 * K) * hd).bfloat16().to(DEV)
    meta = StepMeta(cached, [1] * B)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kc2, vc2, qkv2 = kc.clone(), vc.clone(), qkv.clone()
    ops.rope_cache_write(qkv2, B, i32(list(range(B))), i32(cached), meta.seq_slot, inv_freq, kc2, vc2, table, max_pages, page, H, K, hd,
                         hd, False, True, None, 0, 0)

    class View:
        pass
    view = View()
    view.k, view.v, view.page_table, view.max_pages, view.page_size = kc, vc, table, max_pages, page
    out = torch.full((B + 1, H * hd), 9.0, device=DEV, dtype=torch.bfloat16)
    ops_tensor._device_state(torch.device(DEV)).scratch.fill_(float("nan"))
    scale = 1.0 / math.sqrt(hd)
    ops_tensor.attention_decode_rotary(meta, qkv, view, out, H, K, hd, 0, scale, inv_freq, hd, False, splits=splits, chunk_keys=keys)
    ops_tensor.check_status(torch.device(DEV))
    assert torch.equal(kc.view(torch.int16), kc2.view(torch.int16)) and torch.equal(vc.view(torch.int16), vc2.view(torch.int16))
    for s, n in enumerate(lens):
        pg = int(table[s, (n - 1) // page])
        dense[s][0][n - 1], dense[s][1][n - 1] = kc2[pg, (n - 1) % page].cpu(), vc2[pg, (n - 1) % page].cpu()
    want = reference_attention(qkv2[:, :H * hd].double().cpu().reshape(B, H, hd), dense, list(range(B)), cached, scale, 0)
    close(out[:B], want, 2e-2, 2e-2)
    assert bool((out[B:] == 9.0).all())


def _decode(H, K, hd, cached, splits, fill, st=None):
    """One token for each sequence over filled pages (`fill(keys, values)` changes them first); the pages' plain decode form."""
    from mdma_b200 import ops_tensor
    from test_kernels import DEV, StepMeta, fill_cache
    page, B = 64, len(cached)
    kc, vc, table, max_pages, _ = fill_cache([c + 1 for c in cached], K, hd, page, torch.bfloat16, seed=hd, poison=False)
    fill(kc, vc, table)

    class View:
        pass
    view = View()
    view.k, view.v, view.page_table, view.max_pages, view.page_size = kc, vc, table, max_pages, page
    g = torch.Generator(device=DEV).manual_seed(5)
    qkv = torch.rand(B, (H + 2 * K) * hd, device=DEV, generator=g).bfloat16()
    out = torch.full((B, H * hd), 9.0, device=DEV, dtype=torch.bfloat16)
    ops_tensor.attention(StepMeta(cached, [1] * B), qkv, view, out, H, K, hd, 0, 1.0 / math.sqrt(hd), splits=splits, st=st)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("B", [1, 120])
def test_a_value_that_is_not_finite_shows_however_small_its_share(B, splits):
    """A key whose weight underflows beside another warp's: 0 times infinity is not a number, here as anywhere."""
    def fill(k, v, table):
        k.zero_()
        k[table[0, 0].item(), 0] = 1e4                          # a score of tens of thousands beside zeros
        v[table[0, 1].item(), 7] = float("inf")
    out = _decode(4, 2, 64, [127] * B, splits, fill)
    assert not torch.isfinite(out[0]).any() and torch.isfinite(out[1:]).all()


@pytest.mark.gpu
def test_partial_sums_on_a_boundary_of_four_bytes():
    """Scratch is any array of floats: an odd one gives the bits of an even one."""
    from mdma_b200 import ops_tensor
    from test_kernels import DEV
    outs = []
    for first in (0, 1):
        st = ops_tensor.TensorState(torch.device(DEV), 0, scratch=torch.full((6 * 8 * 3 * 66 + 1,), float("nan"), device=DEV)[first:])
        outs.append(_decode(8, 2, 64, [0, 63, 64, 200, 129, 31], 3, lambda *pages: None, st))
        ops_tensor.check_status(torch.device(DEV), st)
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])


@pytest.mark.gpu
@pytest.mark.parametrize("leaves,launches", [(0, 1), (7, 2)])
def test_a_sequence_keeps_its_bits_when_a_batch_mate_leaves(leaves, launches):
    """The choice that the kernel's caller makes itself, on its own and replayed, around the edges of pieces of 2,048 keys: the
    mate with the longest context leaves (one piece is left, no merge), or a short one (as many pieces)."""
    from mdma_b200 import ops_tensor
    from mdma_b200.parts.rotary import inverse_frequencies
    from test_kernels import DEV, StepMeta, fill_cache, reference_attention
    H = K = 32
    hd, page = 64, 64
    cached = [3000, 2046, 2047, 1500, 31, 1023, 0, 700]         # 2,047 cached and the new token fill a piece
    kc0, vc0, table, max_pages, dense = fill_cache([c + 1 for c in cached], K, hd, page, torch.bfloat16, seed=3)
    inv_freq = inverse_frequencies(hd, 10000.0).to(DEV)
    g = torch.Generator().manual_seed(9)
    rows = torch.randn(len(cached), (H + 2 * K) * hd, generator=g).bfloat16().to(DEV)
    st = ops_tensor.TensorState(torch.device(DEV), ops_tensor.scratch_floats_bound(148, 8, 8, [(H, K, hd)]))

    class View:
        pass

    def run(stay, replay):
        live, mine = [cached[s] for s in stay], rows[stay].contiguous()
        view = View()
        view.k, view.v, view.page_table, view.max_pages, view.page_size = kc0.clone(), vc0.clone(), table[stay].contiguous(), max_pages, page
        meta = StepMeta(live, [1] * len(live))
        meta.most_seqs, meta.most_len, meta.max_len = 8, 3072, -(-(max(live) + 1) // 1024) * 1024
        assert len(live) * K >= st.sms
        out = torch.full((len(live), H * hd), 9.0, device=DEV, dtype=torch.bfloat16)
        step = lambda: ops_tensor.attention_decode_rotary(meta, mine, view, out, H, K, hd, 0, hd ** -0.5, inv_freq, hd, False, st=st)  # noqa: E731
        before = ops_tensor.ops.LAUNCHES
        step()
        count = ops_tensor.ops.LAUNCHES - before
        if replay:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step()
            out.fill_(9.0)
            graph.replay()
            torch.cuda.synchronize()
        ops_tensor.check_status(torch.device(DEV), st)
        return out, count

    everyone = list(range(len(cached)))
    rest = [s for s in everyone if s != leaves]
    with_mate, two = run(everyone, False)
    without, count = run(rest, False)
    assert two == 2 and count == launches                       # pieces and their merge
    assert torch.equal(with_mate[rest], without)
    assert torch.equal(run(everyone, True)[0], with_mate) and torch.equal(run(rest, True)[0], without)
    from mdma_b200 import ops
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kc, vc, turned = kc0.clone(), vc0.clone(), rows.clone()
    B = len(cached)
    ops.rope_cache_write(turned, B, i32(list(range(B))), i32(cached), i32(list(range(B))), inv_freq, kc, vc, table, max_pages, page, H, K, hd,
                         hd, False, True, None, 0, 0)
    for s, c in enumerate(cached):
        pg = int(table[s, c // page])
        dense[s][0][c], dense[s][1][c] = kc[pg, c % page].cpu(), vc[pg, c % page].cpu()
    want = reference_attention(turned[:, :H * hd].double().cpu().reshape(B, H, hd), dense, list(range(B)), cached, hd ** -0.5, 0)
    assert bool(((with_mate.double().cpu() - want.reshape(B, -1)).abs() <= 2e-2 * (1 + want.reshape(B, -1).abs())).all())
