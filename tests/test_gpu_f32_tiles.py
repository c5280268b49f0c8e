"""The float32 kernels for many rows: the bits of the kernels for few rows, which the library's other tests hold to the
plain implementations."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# prompts that end inside and at a tile of 32 queries and of 128 keys, one token, later pieces, several sequences; chunks
# smaller than, equal to and across a tile; grouped heads, a sink, a soft cap, pages of another size
@pytest.mark.parametrize("starts,new,window,heads,dim,page,sink,cap", [
    ([0], [2], (0, 0), (2, 1), 128, 64, False, 0.0), ([0], [32], (0, 0), (2, 2), 64, 64, True, 0.0),
    ([0], [129], (0, 0), (4, 2), 128, 64, False, 5.0), ([0, 0], [300, 33], (0, 0), (4, 1), 64, 16, False, 0.0),
    ([250, 0], [70, 1], (0, 0), (2, 1), 128, 64, True, 0.0), ([0], [300], (1, 20), (2, 1), 64, 64, False, 0.0),
    ([0], [300], (1, 128), (2, 1), 128, 64, True, 0.0), ([90], [290], (1, 100), (2, 2), 64, 64, False, 3.0)])
def test_attention_tiles_give_the_bits_of_the_general_kernel(starts, new, window, heads, dim, page, sink, cap):
    from cpi_b200.csrc import lib as K
    from cpi_b200.engine.batch import BatchStager
    blocks = [-(-(s + n) // page) for s, n in zip(starts, new)]
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(1)).int()
    table = torch.zeros(len(new), max(blocks), dtype=torch.int32)
    at = 0
    for i, b in enumerate(blocks):
        table[i, :b] = order[at:at + b]
        at += b
    stager = BatchStager(DEV)
    batch = stager.stage(list(range(len(new))), starts, [[0] * n for n in new], [[] for _ in new], torch.float32)
    g = torch.Generator(device=DEV).manual_seed(3)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    H, G = heads
    q, k, v = randn(sum(new), H * dim), randn(len(order), G, page, dim), randn(len(order), G, page, dim)
    for i, b in enumerate(blocks):                           # what lies behind a sequence's newest position is not read
        end = starts[i] + new[i] - 1
        k[table[i, end // page].item(), :, end % page + 1:] = float("nan")
        v[table[i, end // page].item(), :, end % page + 1:] = float("nan")
    table = table.to(DEV)
    kw = dict(n_heads=H, n_kv_heads=G, head_dim=dim, window_kind=window[0], window_size=window[1], scale=dim ** -0.5,
              sink=randn(H) if sink else None, softcap=cap)
    want, got = torch.empty_like(q), torch.full_like(q, float("nan"))
    K.attention_general(q, want, k, v, table, page, batch.token_seq, batch.token_pos, batch.seq_slot, **kw)
    K.attention_f32_tiles(q, got, k, v, table, page, batch, **kw)
    assert bool(want.isfinite().all()) and torch.equal(got, want)


# both tile widths (64 and 128 weight rows), edges of both, K that is no multiple of 16 or 4, unaligned rows, groups of unequal
# rows (one empty), a row gather and scatter, every mode and pair of types
@pytest.mark.parametrize("M,N,K", [(64, 64, 16), (65, 129, 50), (200, 30, 7), (130, 4100, 64), (17, 1, 129), (700, 2056, 33)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4, 5, 6])
def test_products_of_many_rows_give_the_bits_of_the_kernel_for_few(M, N, K, mode):
    from cpi_b200.csrc import lib as L
    g = torch.Generator(device=DEV).manual_seed(M + mode)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    glu = mode in L.GATED_MODES
    types = [(torch.float32, torch.float32, torch.float32), (torch.float32, torch.bfloat16, torch.float32),
             (torch.bfloat16, torch.bfloat16, torch.bfloat16 if mode != 1 else torch.float32)]
    for i, (ta, tw, to) in enumerate(types):
        off = i % 2                                          # rows that do not start on 16 bytes
        a = randn(M + 5, K + 4 * off + off).to(ta)[:, off:off + K]
        groups = 3
        w = (randn(groups, (2 if glu else 1) * N, K) * 0.1).to(tw)
        rows = torch.randperm(M + 5, generator=g, device=DEV)[:M].int()
        cut = M // 3
        offsets = torch.tensor([0, cut, cut, M], dtype=torch.int32, device=DEV)
        scale = randn(M)
        for kw in (dict(), dict(a_rows=rows, group_offsets=offsets, n_groups=groups, row_scale=scale, out_rows=rows)):
            ww = w if kw else w[0]
            outs = []
            for hint in (16, 64):
                out = torch.linspace(-1, 1, (M + 5) * N, device=DEV).view(M + 5, N).to(to)
                L.gemm_simt(a, ww, out, mode, m_rows=M, rows_per_group_hint=hint, gate_limit=0.7, **kw)
                outs.append(out)
            assert torch.equal(outs[0], outs[1]) and bool(outs[0].isfinite().all())


# the choice between the two kernels: a sliding window as long as the longest context and one shorter, chunks, a score cap, kept first
# positions, heads of another size; rows off 16 bytes, which only the general kernel takes
@pytest.mark.parametrize("starts,new,window,size,keep,dim,off,tiles", [
    ([0], [150], "full", 0, 0, 64, 0, True), ([70, 0], [60, 9], "sliding", 130, 0, 64, 0, True), ([70, 0], [60, 9], "sliding", 129, 0, 64, 0, False),
    ([0, 30], [90, 70], "sliding", 64, 5, 128, 0, False), ([0, 30], [90, 70], "sliding", 100, 5, 128, 0, True),
    ([20, 0], [90, 70], "chunk", 48, 0, 128, 0, True), ([0], [70], "full", 0, 0, 32, 0, False), ([0], [70], "full", 0, 0, 64, 1, False),
    ([40, 9], [1, 1], "full", 0, 0, 64, 0, False)])
def test_both_routes_of_float32_attention_give_the_same_bits(starts, new, window, size, keep, dim, off, tiles, monkeypatch):
    from cpi_b200.csrc import lib as K
    from cpi_b200.engine.batch import BatchStager
    from cpi_b200.parts import attention
    blocks = max(-(-(s + n) // 64) for s, n in zip(starts, new))
    table = torch.arange(len(new) * blocks, dtype=torch.int32, device=DEV).flip(0).view(len(new), blocks)
    stager = BatchStager(DEV)
    batch = stager.stage(list(range(len(new))), starts, [[0] * n for n in new], [[] for _ in new], torch.float32)
    g = torch.Generator(device=DEV).manual_seed(4)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    H, G, T = 4, 2, sum(new)
    q = randn(T * H * dim + off)[off:].view(T, H * dim)
    k, v = randn(len(new) * blocks, G, 64, dim), randn(len(new) * blocks, G, 64, dim)
    calls, tile_kernel = [], K.attention_f32_tiles
    monkeypatch.setattr(K, "attention_f32_tiles", lambda *a, **kw: calls.append(1) or tile_kernel(*a, **kw))
    outs = []
    for use in (True, False):
        monkeypatch.setattr(attention, "use_tile_kernel", use)
        out = torch.full((T, H * dim), float("nan"), device=DEV)
        attention.attend(q, out, k, v, table, 64, batch, n_heads=H, n_kv_heads=G, head_dim=dim, value_dim=dim, window_kind=window,
                         window_size=size, scale=dim ** -0.5, sink=randn(H) * 0 + 0.3, keep_first=keep, softcap=4.0)
        outs.append(out)
        assert len(calls) == int(tiles)
    assert bool(outs[0].isfinite().all()) and torch.equal(outs[0], outs[1])


# the wide tile (many rows and columns; from one and a half CTAs an SM for longer sums, bfloat16 weights from two), either loop of it
# and of the narrow one, and its depths for bfloat16 weights
@pytest.mark.parametrize("M,N,K,mode", [(1500, 2056, 130, 0), (1500, 1028, 131, 2), (2000, 1500, 128, 1), (90, 200, 64, 0), (90, 200, 65, 2), (70, 300, 200, 0),
                                        (1500, 6200, 63, 0), (1500, 3100, 65, 2), (1500, 6200, 129, 1), (2000, 900, 4100, 0), (2000, 900, 2000, 1),
                                        (70, 300, 192, 2), (70, 300, 193, 1), (900, 1000, 385, 0), (900, 1000, 384, 0)])
def test_more_products_of_many_rows_give_the_bits_of_the_kernel_for_few(M, N, K, mode):
    from cpi_b200.csrc import lib as L
    g = torch.Generator(device=DEV).manual_seed(M)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    for tw in (torch.float32, torch.bfloat16):
        a, w = randn(M, K), randn(N * (2 if mode == 2 else 1), K).to(tw)
        start = randn(M, N)
        got = start.clone()
        L.gemm_simt(a, w, got, mode)
        for r in range(0, M, 16 * 37):                       # sixteen rows at a time take the kernel for few
            want = start[r:r + 16].clone()
            L.gemm_simt(a[r:r + 16], w, want, mode)
            assert torch.equal(got[r:r + 16], want), (tw, r)
