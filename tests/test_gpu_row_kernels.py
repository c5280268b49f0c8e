"""Row kernels with more than one route: the vectorised convolution, the warp-sized gated norm, the choice and the lists of
routed experts, and products whose features are no multiple of the two-SM kernel's tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device=DEV)


# one and eight tokens a thread (by the number of blocks), sequence ends inside a thread's run, steps shorter than the taps
@pytest.mark.parametrize("taps", [1, 2, 4, 8])
@pytest.mark.parametrize("new,channels", [([1, 1, 1], 12), ([3, 2, 40], 516), ([309, 1, 9, 7], 4100)])
def test_convolution_routes_give_the_same_bits(taps, new, channels):
    from cpi_b200.csrc import lib as K
    from cpi_b200.engine.batch import BatchStager
    randn = _rand(taps)
    T, B = sum(new), len(new)
    stager = BatchStager(DEV)
    batch = stager.stage(list(range(B)), [5] * B, [[0] * n for n in new], [[]] * B, torch.float32)
    x, w, b, ib = randn(T, channels + 4), randn(channels, taps), randn(channels), randn(channels)
    wide = torch.zeros(T, channels + 5, device=DEV)
    wide[:, 1:] = x                                          # the same rows off their 16 bytes: the kernel without vectors
    carry = randn(B, max(taps - 1, 0), channels)
    outs = []
    for rows in (x[:, 4:], wide[:, 5:]):
        c, out = carry.clone(), torch.empty(T, channels, device=DEV)
        K.causal_conv(rows, w, b, c, out, batch, silu=True, in_bias=ib)
        outs.append((out, c))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("n", [4, 100, 128, 132, 256, 260, 512, 516, 1020, 1024])
@pytest.mark.parametrize("first,act,shared", [(True, "silu", False), (False, "sigmoid", True), (False, "silu", False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_norm_of_every_width(n, first, act, shared, dtype):
    from cpi_b200.csrc import lib as K
    randn, T, parts = _rand(n), 7, 3
    y, gate, w = randn(T, parts * n), randn(T, parts * n + 4)[:, 4:], randn(n if shared else parts * n)
    out = torch.empty(T, parts * n, device=DEV, dtype=dtype)
    K.gated_norm(y, gate, w, out, parts=parts, gate_first=first, eps=1e-5, gate_act=act)
    g = torch.sigmoid(gate.double()) * (gate.double() if act == "silu" else 1.0)
    v = (y.double() * g if first else y.double()).view(T, parts, n)
    ref = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)) * w.double().view(-1, n)
    ref = ref.reshape(T, -1) * (1.0 if first else g)
    # float32: the sum of n squares and a dozen operations; bfloat16: one rounding to 8 bits more
    tol = 2.0 ** -19 if dtype == torch.float32 else 2.0 ** -8 * 1.01
    assert bool(((out.double() - ref).abs() <= tol * ref.abs() + 2.0 ** -21 * ref.abs().max()).all())


@pytest.mark.parametrize("experts,top_k", [(1, 1), (16, 4), (33, 33), (256, 8), (40, 35)])
@pytest.mark.parametrize("mode", [False, True, "softmax_chosen"])
def test_choice_of_experts_with_ties_and_nan(experts, top_k, mode):
    from cpi_b200.csrc import lib as K
    T, randn = 70, _rand(experts)
    logits = (randn(T, experts) * 2).round() / 2             # many ties
    logits[3] = float("nan")
    logits[4, ::2] = float("nan")
    logits[5] = float("-inf")
    logits[6, 0] = -0.0
    idx, gate = torch.empty(T, top_k, dtype=torch.int32, device=DEV), torch.empty(T, top_k, device=DEV)
    K.router_select(logits, idx, gate, top_k=top_k, sigmoid_gate=mode)
    for t, row in enumerate(logits.tolist()):
        order = sorted((e for e in range(experts) if row[e] == row[e]), key=lambda e: (-row[e], e))
        order += [e for e in range(experts) if row[e] != row[e]]
        assert idx[t].tolist() == order[:top_k]
        chosen = torch.tensor([row[e] for e in order[:top_k]], dtype=torch.float64)
        want = torch.ones(top_k, dtype=torch.float64) if mode is False else torch.sigmoid(chosen) if mode is True \
            else torch.softmax(chosen, 0)
        got = gate[t].double().cpu()
        assert torch.equal(got.isnan(), want.isnan())
        assert float((got - want).nan_to_num().abs().max()) <= 2.0 ** -20


@pytest.mark.parametrize("T,top_k,experts", [(1, 1, 1), (700, 3, 20), (2048, 4, 16), (9000, 2, 256)])
def test_expert_lists_are_stable(T, top_k, experts):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(T)
    idx = torch.randint(0, experts, (T, top_k), generator=g, device=DEV, dtype=torch.int32)
    gate = torch.rand(T, top_k, generator=g, device=DEV)
    i32 = lambda n: torch.empty(n, dtype=torch.int32, device=DEV)
    offsets, token, slot, scale = i32(experts + 1), i32(T * top_k), i32(T * top_k), torch.empty(T * top_k, device=DEV)
    K.moe_lists(idx, gate, offsets, token, scale, slot, n_tokens=T, top_k=top_k, n_experts=experts)
    flat = idx.view(-1).long()
    order = torch.sort(flat, stable=True).indices
    assert torch.equal(token.long(), order // top_k) and torch.equal(scale, gate.view(-1)[order])
    assert torch.equal(slot.long()[order], torch.arange(T * top_k, device=DEV))
    assert offsets.tolist() == [0] + torch.bincount(flat, minlength=experts).cumsum(0).tolist()


# features past the last pair's first half, inside its second half, one more than a whole tile, odd (direct epilogue); a token
# tile that ends early
@pytest.mark.parametrize("N", [1025, 1100, 1344, 1480, 1536 + 8])
@pytest.mark.parametrize("mode,out_dtype", [(0, torch.float32), (0, torch.bfloat16), (1, torch.float32), (2, torch.bfloat16), (5, torch.bfloat16)])
def test_two_sm_products_of_any_number_of_features(N, mode, out_dtype):
    from cpi_b200.csrc import lib as K
    randn, T, Kd = _rand(N + mode), 700, 264
    a, w = randn(T, Kd).bfloat16(), (randn((2 if mode == 2 else 1) * N, Kd) * 0.1).bfloat16()
    out = randn(T, N + 8).to(out_dtype)
    before = out.clone()
    assert K.gemm_tc_pair(a, w, out[:, :N], mode, any_features=True)
    acc = a.double() @ w.double().T
    if mode == 2:
        ref = torch.nn.functional.silu(acc[:, :N]) * acc[:, N:]
    else:
        ref = torch.relu(acc) ** 2 if mode == 5 else acc + (before[:, :N].double() if mode == 1 else 0.0)
    # float32 sums of 264 products in the tensor cores' order, and the output's rounding
    tol = 2.0 ** -16 if out_dtype == torch.float32 else 2.0 ** -8 * 1.02
    assert bool(((out[:, :N].double() - ref).abs() <= tol * ref.abs() + 2.0 ** -14 * ref.abs().max() * 0.1).all())
    assert torch.equal(out[:, N:], before[:, N:]) and int(K.tc_error_flag(DEV)) == 0


@pytest.mark.parametrize("T,N,Kd,mode,pays", [
    (2048, 1288, 2048, 0, False), (2048, 3144, 2048, 0, True), (1024, 4104, 2048, 1, False), (1024, 1032, 2048, 0, True),
    (1024, 1032, 8192, 0, False), (512, 1032, 4096, 0, False), (8192, 1032, 512, 0, False), (700, 1025, 264, 0, False),
    (2048, 4104, 512, 2, True), (4096, 1160, 512, 2, False), (512, 1544, 512, 2, True), (511, 10304, 512, 0, False)])
def test_features_that_are_no_multiple_take_the_faster_kernel(T, N, Kd, mode, pays, monkeypatch):
    """Both sides of the rule on a GPU of 148 SMs, and that a product asks it."""
    from cpi_b200.csrc import lib as K
    from cpi_b200.parts import linear
    if K.sm_count() != 148:
        pytest.skip("the rule counts waves of 148 SMs")
    assert K.gemm_tc_pair_pays(T, N, Kd, mode == 2) == pays
    taken, pair = [], K.gemm_tc_pair
    monkeypatch.setattr(K, "gemm_tc_pair", lambda *a, **kw: taken.append(pair(*a, **kw)) or taken[-1])
    randn = _rand(N)
    a, w = randn(T, Kd).bfloat16(), (randn((2 if mode == 2 else 1) * N, Kd) * 0.1).bfloat16()
    out = torch.zeros(T, N, device=DEV, dtype=torch.bfloat16 if mode == 2 else torch.float32)
    linear.project(a, w, out, mode)
    assert taken == ([] if T < 512 else [pays])
    rows = torch.tensor([0, T // 2, T - 1], device=DEV)
    acc = a[rows].double() @ w.double().T
    ref = torch.nn.functional.silu(acc[:, :N]) * acc[:, N:] if mode == 2 else acc
    # float32 sums of Kd products in the tensor cores' order, and the output's rounding
    tol = 2.0 ** -8 * 1.02 if mode == 2 else 2.0 ** -16
    assert bool(((out[rows].double() - ref).abs() <= tol * ref.abs() + 2.0 ** -14 * ref.abs().max() * 0.1).all())
