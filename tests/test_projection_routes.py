"""What `project` hands to the kernels: every keyword argument reaches the one that is asked, which refuses what it does not take."""
import pytest
import torch

from cpi_b200.csrc import lib as K
from cpi_b200.parts import linear


def _operands(groups=2, T=3):
    a, w = torch.zeros(groups * T, 16, dtype=torch.bfloat16), torch.zeros(groups, 8, 16, dtype=torch.bfloat16)
    offsets = torch.arange(groups + 1, dtype=torch.int32) * T
    return a, w, torch.zeros(groups * T, 8), dict(group_offsets=offsets, n_groups=groups, rows_per_group_hint=T)


@pytest.mark.parametrize("extra", [{}, {"row_scale": torch.ones(6)}, {"a_rows": torch.arange(6)}, {"m_rows": 6}, {"gate_limit": 2.0},
                                   {"out_rows": torch.arange(6)}])
def test_products_of_even_groups_lose_no_argument(monkeypatch, extra):
    a, w, out, groups = _operands()
    asked = []
    monkeypatch.setattr(K, "gemm_few", lambda *args, **kw: asked.append(kw) or True)
    linear.project(a, w, out, even_groups=2, **groups, **extra)
    assert len(asked) == 1 and asked[0]["even_groups"] == 2
    assert all(asked[0].get(name) is value for name, value in extra.items())


@pytest.mark.parametrize("extra", [{"row_scale": torch.ones(6)}, {"a_rows": torch.arange(6)}, {"n_out": 8}, {"n_groups": 3}])
def test_what_products_of_even_groups_leave_to_other_kernels(extra):
    a, w, out, groups = _operands()
    assert not K.gemm_few(a, w, out, even_groups=2, **{**groups, **extra})


def test_a_product_may_be_kept_from_the_kernel_for_a_handful_of_tokens(monkeypatch):
    a, w, out = torch.zeros(4, 16, dtype=torch.bfloat16), torch.zeros(8, 16, dtype=torch.bfloat16), torch.zeros(4, 8)
    asked = []
    monkeypatch.setattr(K, "gemm_few", lambda *args, **kw: asked.append("few") or True)
    monkeypatch.setattr(K, "gemm_tc", lambda *args, **kw: asked.append("tc") or "few" not in kw)
    linear.project(a, w, out)
    linear.project(a, w, out, few=False)
    assert asked == ["few", "tc"]
