"""Attention of single tokens over cached latent rows, by teams of warps (csrc/latent_attention.cu), and the rows' norms of one
launch (csrc/latent.cu), against plain computations in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda:0", 64


# one and two row groups of heads, up to and over the tiles of 32 that the teams hold at once, one and two tiles a team,
# contexts that end at a tile's and a page's edge, windows, keys whole and divided, a sink; more than 32 heads
@pytest.mark.parametrize("H,rank,rot,lens,splits,window,sink", [
    (1, 16, 16, [1, 32, 33], 1, 0, False), (16, 512, 64, [1500, 64], 1, 0, True), (16, 512, 64, [2001, 129], 5, 0, False),
    (8, 256, 64, [700, 65, 1], 2, 0, True), (24, 512, 64, [900, 31], 2, 0, False), (32, 512, 128, [640, 257], 1, 300, True),
    (17, 64, 16, [500, 128], 3, 100, False), (16, 256, 64, [4000], 40, 0, False), (40, 128, 32, [300, 96], 2, 0, True)])
def test_single_tokens(H, rank, rot, lens, splits, window, sink):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(3)
    row, T = rank + rot, len(lens)
    blocks = [-(-n // PAGE) for n in lens]
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(1)).int()
    table, at = torch.zeros(T, max(blocks), dtype=torch.int32), 0
    cache = torch.full((sum(blocks), 1, PAGE, row), float("nan"), dtype=torch.bfloat16, device=DEV)     # nothing behind the newest position is read
    rows = []
    for i, (n, b) in enumerate(zip(lens, blocks)):
        table[i, :b] = order[at:at + b]
        at += b
        x = torch.randn(n, row, generator=g, device=DEV).bfloat16() * 0.7
        rows.append(x)
        for j in range(b):
            cache[table[i, j].item(), 0, :min(PAGE, n - j * PAGE)] = x[j * PAGE:(j + 1) * PAGE]
    q = torch.randn(T, H * row, generator=g, device=DEV).bfloat16()
    snk = torch.randn(H, generator=g, device=DEV) if sink else None
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out = torch.full((H * T, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.latent_attention(q, out, cache, table.to(DEV), PAGE, i32(list(range(T))), i32([n - 1 for n in lens]), i32(list(range(T))), n_heads=H,
                       rank=rank, scale=row ** -0.5, sink=snk, n_splits=splits, window=window)
    for t, x in enumerate(rows):
        keys = x.double()[-window if window else 0:]
        s = q[t].double().view(H, row) @ keys.T * row ** -0.5
        if snk is not None:
            s = torch.cat([s, snk.double()[:, None]], 1)
        ref = torch.softmax(s, -1)[:, :keys.shape[0]] @ keys[:, :rank]
        got = out.view(H, T, rank)[:, t].double()
        # probabilities and the result are rounded to bfloat16 (2^-9 each of values up to the largest)
        assert (got - ref).norm() <= 2.0 ** -7 * ref.norm() and (got - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()


@pytest.mark.parametrize("T,rank,rot,q_rank,dtype", [(1, 512, 64, 768, torch.bfloat16), (70, 96, 32, 30, torch.bfloat16), (5, 512, 64, 5000, torch.float32),
                                                     (9, 61, 2, 64, torch.float32)])
def test_both_norms_of_one_launch(T, rank, rot, q_rank, dtype):
    """The latent into its page and the queries' latent beside it, rows in fours and one by one."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(T, q_rank + rank + rot, generator=g, device=DEV)
    w1, w2 = torch.randn(rank, generator=g, device=DEV), torch.randn(q_rank, generator=g, device=DEV)
    pages = -(-T // PAGE)
    cache = torch.zeros(pages, 1, PAGE, rank + rot, dtype=dtype, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cq = torch.zeros(T, q_rank, dtype=dtype, device=DEV)
    K.latent_kv_write(x[:, q_rank:], w1, 1e-6, None, False, cache, i32([list(range(pages))]), PAGE, i32([0] * T), i32(list(range(T))), i32([0]),
                      rank=rank, rot=rot, queries=(x[:, :q_rank], w2, cq))
    norm = lambda v, w: v.double() / torch.sqrt((v.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20)
    for got, ref in ((cache.view(-1, rank + rot)[:T, :rank], norm(x[:, q_rank:q_rank + rank], w1)), (cq, norm(x[:, :q_rank], w2))):
        assert ((got.double() - ref).abs() <= tol * ref.abs() + 1e-30).all()
    assert torch.equal(cache.view(-1, rank + rot)[:T, rank:], x[:, q_rank + rank:].to(dtype))
