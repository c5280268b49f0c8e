"""The product for a handful of tokens (csrc/gemm_few.cu) against 64-bit products: edges of its 16 features, 8 tokens and 32 k."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from cpi_b200.csrc import lib
    return lib


def operands(T, N, Kd, rows, seed=0, ldx=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randn(T, Kd + ldx, generator=g, device=DEV).bfloat16()[:, :Kd]
    w = torch.randn(rows, Kd, generator=g, device=DEV).bfloat16()
    return a, w


def bound(a, w, out):
    """Products of bfloat16 pairs are exact in float32; a sum of K of them in any order is off by at most K + 1 truncations."""
    return (a.shape[1] + 1) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T) + 1e-30


def launch(a, w, out, mode, form, limit=0.0):
    from ctypes import c_float, c_int, c_long
    k = K()
    k._call("cpi_gemm_few", k._p(a), c_long(a.stride(0)), k._p(w), k._p(out), c_int(k.dtype_code(out.dtype)), c_long(out.stride(0)),
            k._p(None), c_int(1), c_int(a.shape[0]), c_int(out.shape[1]), c_int(a.shape[1]), c_int(mode), c_int(form), c_float(limit), k._stream())


@pytest.mark.parametrize("form", [1, 2, 3, 4])
@pytest.mark.parametrize("T,N,Kd", [(1, 1, 8), (1, 17, 40), (3, 520, 264), (8, 16, 1032), (9, 33, 2048), (16, 200, 4104), (2, 48, 8200)])
def test_forms_against_64_bit_products(form, T, N, Kd):
    k = K()
    a, w = operands(T, N, Kd, N, ldx=24)
    ref = a.double() @ w.double().T
    for dt in (torch.float32, torch.bfloat16):
        buf = torch.full((T + 1, N + 5), 7.0, device=DEV, dtype=dt)
        out = buf[:T, :N]
        launch(a, w, out, k.MODE_STORE, form)
        tol = bound(a, w, out) + (2.0 ** -8 * ref.abs() if dt == torch.bfloat16 else 0)
        assert ((out.double() - ref).abs() <= tol).all()
        assert (buf[T] == 7).all() and (buf[:, N:] == 7).all()                  # nothing beside the outputs
    res = torch.randn(T, N, device=DEV)
    out = res.clone()
    launch(a, w, out, k.MODE_ADD, form)
    assert ((out.double() - res.double() - ref).abs() <= bound(a, w, out) + 2.0 ** -23 * out.double().abs()).all()


@pytest.mark.parametrize("T,N,Kd", [(17, 200, 264), (24, 2368, 520), (32, 16, 2048), (32, 33, 8)])
def test_more_tokens(T, N, Kd):
    k = K()
    a, w = operands(T, N, Kd, N)
    out = torch.zeros(T, N, device=DEV)
    assert k.gemm_few(a, w, out) == (N <= 16 * k.sm_count())
    if N <= 16 * k.sm_count():
        assert ((out.double() - a.double() @ w.double().T).abs() <= bound(a, w, out)).all()


@pytest.mark.parametrize("T", [1, 8, 11, 32])
def test_gates_and_activations(T):
    """Every mode against the tcgen05 kernel's epilogue: the same functions of sums that agree to the order of their terms."""
    k = K()
    N, Kd = 72, 512
    a, w = operands(T, N, Kd, 2 * N, seed=3)
    w *= 0.05
    forms = [1] if T > 16 else [1, 2, 3, 4]
    for mode in (k.MODE_SWIGLU, k.MODE_GEGLU, k.MODE_CLAMPED_GLU, k.MODE_STORE_RELU2, k.MODE_STORE_GELU):
        gated = mode in k.GATED_MODES
        wm = w if gated else w[:N].contiguous()
        want, limit = torch.zeros(T, N, device=DEV, dtype=torch.bfloat16), 2.0 if mode == k.MODE_CLAMPED_GLU else 0.0
        assert k.gemm_tc(a, wm, want, mode, gate_limit=limit)
        for form in forms:
            got = torch.zeros_like(want)
            launch(a, wm, got, mode, form, limit)
            # (a bfloat16 step, where a sum's last bits tip the rounding, and what sums near zero differ by)
            assert ((got - want).float().abs() <= 2.0 ** -7 * want.float().abs() + 1e-4).all(), (mode, form)


def test_what_it_leaves_to_other_kernels():
    k = K()
    a, w = operands(4, 64, 128, 64)
    out = torch.zeros(4, 64, device=DEV)
    assert k.gemm_few(a, w, out)
    assert not k.gemm_few(a.float(), w, out) and not k.gemm_few(a, w.float(), out)
    assert not k.gemm_few(a[:, 4:], w[:, 4:], out)                                # rows off 16 bytes
    assert not k.gemm_few(a, w, out, k.MODE_SWIGLU) and not k.gemm_few(a, w, out.bfloat16(), k.MODE_ADD)
    assert not k.gemm_few(a, w, out, row_scale=torch.ones(4, device=DEV))
    assert not k.gemm_few(operands(33, 64, 128, 64)[0], w, torch.zeros(33, 64, device=DEV))


@pytest.mark.parametrize("groups,T,N,Kd", [(3, 1, 17, 40), (16, 8, 512, 128), (16, 8, 128, 512), (5, 16, 64, 264), (2, 9, 33, 8)])
def test_even_groups(groups, T, N, Kd):
    """Every group's rows by its own weights, sent where the row list says."""
    k = K()
    a, _ = operands(groups * T, N, Kd, 1, ldx=8)
    w = torch.randn(groups, N, Kd, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).bfloat16()
    rows = torch.randperm(groups * T, generator=torch.Generator().manual_seed(2)).int().to(DEV)
    ref = torch.einsum("gtk,gnk->gtn", a.double().view(groups, T, Kd), w.double()).reshape(groups * T, N)
    tol = torch.einsum("gtk,gnk->gtn", a.double().abs().view(groups, T, Kd), w.double().abs()).reshape(groups * T, N) * (Kd + 1) * 2.0 ** -23 + 1e-30
    for to in (None, rows):
        buf = torch.full((groups * T, N + 3), 7.0, device=DEV)
        assert k.gemm_few(a, w, buf[:, :N], even_groups=groups, out_rows=to)
        got = buf[:, :N] if to is None else buf[rows.long()][:, :N]
        assert ((got.double() - ref).abs() <= tol).all() and (buf[:, N:] == 7).all()
    assert not k.gemm_few(a, w, buf[:, :N], even_groups=groups + 1)


@pytest.mark.parametrize("T,per_sm,Kd,gated,takes", [
    (1, 13.5, 256, False, False), (1, 13.5, 2048, False, True), (8, 7, 128, False, False), (1, 13.5, 1024, True, False), (4, 3.9, 16384, False, True),
    (16, 2.1, 8192, False, False), (16, 2.1, 2048, False, True), (16, 2.1, 4096, True, False), (9, 1.5, 8192, False, True), (9, 1.5, 12288, False, False),
    (32, 0.4, 8192, False, False), (17, 0.4, 8192, False, True), (17, 0.1, 8192, True, False), (17, 0.9, 4096, True, True), (16, 0.9, 16384, True, True)])
def test_products_that_gemm_tc_finishes_sooner_are_left_to_it(T, per_sm, Kd, gated, takes):
    """Blocks of 16 features per SM, the depth and the tokens decide (the times of both sides stand at the rule)."""
    k = K()
    N = 16 * int(per_sm * k.sm_count())
    assert bool(k._plan("few", torch.cuda.current_device(), T, N, Kd, 0, gated)) == takes
    if not takes:                                                             # (asked with operands as well: refused before they are read)
        a = torch.zeros(T, Kd, device=DEV, dtype=torch.bfloat16)
        out = torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
        w = torch.empty(2 * N if gated else N, Kd, device=DEV, dtype=torch.bfloat16)
        assert not k.gemm_few(a, w, out, k.MODE_SWIGLU if gated else k.MODE_STORE)


@pytest.mark.parametrize("T,top,taken", [(1, 1, 0), (2, 1, 0), (1, 2, 0), (4, 1, 2), (2, 2, 2)])
@pytest.mark.parametrize("overlap", [True, False])
def test_a_small_shared_expert_beside_one_or_two_routed_rows(monkeypatch, T, top, taken, overlap):
    """Its two products stay on the tcgen05 kernel then, beside the routed ones and after them alike."""
    from cpi_b200.config.spec import PartSpec
    from cpi_b200.engine.batch import BatchStager
    from cpi_b200.parts import Workspace, build_part
    from cpi_b200.weights import DictSource
    k = K()
    part = build_part("feed_forward", PartSpec("moe_swiglu", {"hidden_size": 256, "num_experts": 8, "top_k": top, "expert_size": 128,
                                                             "shared_size": 128, "router_gate": "softmax_chosen"}), "", workspace=Workspace(DEV))
    g = torch.Generator(device=DEV).manual_seed(1)
    part.load(DictSource({r.name: (torch.randn(*r.shape, generator=g, device=DEV) * 0.05).bfloat16() for r in part.requirements()}), DEV)
    part.overlap_shared = overlap
    calls, real = [], k.gemm_few
    monkeypatch.setattr(k, "gemm_few", lambda *a, **kw: calls.append(real(*a, **kw)) or calls[-1])
    stager = BatchStager(DEV)
    batch = stager.stage(list(range(T)), [0] * T, [[0]] * T, [[]] * T, torch.bfloat16)
    out = torch.zeros(T, 256, device=DEV)
    part.forward(torch.randn(T, 256, generator=g, device=DEV).bfloat16(), out, batch)
    assert sum(calls) == taken and bool(out.isfinite().all()) and bool(out.any())
