"""The row preparation with a warp per head against the general form, which the same rows take when they do not start on 16 bytes."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one token, a few, enough for blocks of whole rows; heads that fill a block's warps and that don't; rotations of nothing, a part
# (ending at the first and at a later lane) and all of a head, in both layouts; norms over nothing, a head, the projection
@pytest.mark.parametrize("T,nh,nkv,d", [(1, 4, 1, 64), (3, 16, 4, 128), (40, 6, 6, 128), (301, 10, 2, 64), (300, 40, 8, 128)])
@pytest.mark.parametrize("rot,interleaved,norm,bias,write", [(0, False, "none", True, True), ("all", False, "whole", True, True),
                                                             ("half", True, "head", False, True), (8, False, "head_weighted", True, True),
                                                             ("half", False, "whole", False, False)])
@pytest.mark.parametrize("src,dst", [("f32", "bf16"), ("f32", "f32"), ("bf16", "bf16")])
def test_heads_equal_the_general_form(T, nh, nkv, d, rot, interleaved, norm, bias, write, src, dst):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(T + d)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    dt = {"f32": torch.float32, "bf16": torch.bfloat16}
    page, n = 16, (nh + 2 * nkv) * d
    rows, i32 = randn(T, n).to(dt[src]), lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    # two sequences, their pages in no order
    first = T // 2
    seq, pos = i32([0] * first + [1] * (T - first)), i32(list(range(first)) + list(range(5, 5 + T - first)))
    blocks = -(-(T + 5) // page)
    table = i32(torch.randperm(2 * blocks, generator=torch.Generator().manual_seed(1)).tolist()).view(2, blocks)
    slot = i32([1, 0])
    rot = {"all": d, "half": d // 2}.get(rot, rot)
    kw = dict(n_heads=nh, n_kv_heads=nkv, head_dim=d, value_dim=d, interleaved=interleaved, write_kv=write, norm_eps=1e-6,
              norm_whole=norm == "whole", head_norm={"head": 1, "head_weighted": 2}.get(norm, 0), temperature=(64.0, 0.1),
              rotary_amplitude=1.1, inv_freq=None if rot == 0 else 1e4 ** (-torch.arange(rot // 2, device=DEV, dtype=torch.float32) * 2 / rot),
              rotary_dims=rot, bias=randn(n) if bias else None)
    if norm in ("whole", "head_weighted"):
        kw.update(q_norm=randn(nh * d if norm == "whole" else d), k_norm=randn(nkv * d if norm == "whole" else d))
    got = []
    for off in (0, 1):                                # a row that starts an element later takes the general form
        x = torch.empty(T, n + 8, dtype=dt[src], device=DEV)[:, off:off + n]
        x.copy_(rows)
        q = torch.full((T, nh * d), 7.0, dtype=dt[dst], device=DEV)
        kc, vc = (torch.full((2 * blocks, nkv, page, d), 7.0, dtype=dt[dst], device=DEV) for _ in range(2))
        K.qkv_prepare(x, q, kc, vc, table, page, seq, pos, slot, **kw)
        got.append((q, kc, vc))
    # Sums of squares in another order, and products that may be fused otherwise: 2^-21 of an element or (a difference of two
    # turned elements) of the largest.  In bfloat16 that may move a result to its neighbour, which is up to 2^-7 of it away (8
    # bits, a unit of the last of which is 2^-7 of a power of two), where it lies that near the middle: of 2^-8 steps 2^-12 or so.
    unit = 2.0 ** -7 if dst == "bf16" else 2.0 ** -21
    for a, b in zip(*got):
        a, b = a.double(), b.double()
        assert bool(((a - b).abs() <= unit * b.abs() + 2.0 ** -21 * b.abs().max()).all())
        assert dst == "f32" or float((a != b).double().mean()) <= 2.0 ** -8
    assert write or bool((got[0][1] == 7.0).all() and (got[0][2] == 7.0).all())


@pytest.mark.parametrize("norm", [0, 1])
def test_rows_beyond_shared_memory_are_refused_by_either_form(norm):
    """410 heads of 128 are 205 KB of q and k rows, 200 heads with the rotated rows beside them too: neither form takes them."""
    from cpi_b200.csrc import lib as K
    nh, nkv, d = (200, 5, 128) if norm else (400, 10, 128)
    n = (nh + 2 * nkv) * d
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    for off in (0, 1):
        x = torch.zeros(1, n + 8, device=DEV)[:, off:off + n]
        q = torch.zeros(1, nh * d, device=DEV)
        kc, vc = (torch.zeros(1, nkv, 16, d, device=DEV) for _ in range(2))
        with pytest.raises(K.KernelError, match="does not fit in shared memory"):
            K.qkv_prepare(x, q, kc, vc, i32(0).view(1, 1), 16, i32(0), i32(0), i32(0), n_heads=nh, n_kv_heads=nkv, head_dim=d,
                          value_dim=d, head_norm=norm, norm_eps=1e-6)
