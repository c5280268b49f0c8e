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
