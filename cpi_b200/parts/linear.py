"""Matrix products of the parts: picks the kernel for a contraction out[m, n] = sum_k a[m, k] w[n, k].

bfloat16 activations and weights whose shapes the tensor-core kernels accept go to the tcgen05
kernels, or for a handful of tokens to one that is over when theirs have begun; everything else -- the whole float32 path, mixed dtypes, odd shapes -- goes to the FP32-pipe
kernel, which accepts any size.  Either way accumulation is float32.
"""
from __future__ import annotations

import torch

from ..csrc import lib as K

MODE_STORE, MODE_ADD, MODE_SWIGLU, MODE_GEGLU = K.MODE_STORE, K.MODE_ADD, K.MODE_SWIGLU, K.MODE_GEGLU
MODE_CLAMPED_GLU, MODE_STORE_RELU2, MODE_STORE_GELU = K.MODE_CLAMPED_GLU, K.MODE_STORE_RELU2, K.MODE_STORE_GELU

# set to False to force the FP32-pipe kernel everywhere (tests compare the two)
use_tensor_cores = True
# set to False to keep dense products with many tokens on the single-CTA kernel
use_paired_kernel = True


class single_cta_products:
    """While entered, products with many tokens stay on the single-CTA kernel (a block whose chains of launches the
    two-SM kernel is not cleared for wraps its sublayers in this).  Host-side routing only; nests."""
    depth = 0

    def __enter__(self):
        single_cta_products.depth += 1

    def __exit__(self, *exc):
        single_cta_products.depth -= 1


def project(a, w, out, mode=MODE_STORE, *, even_groups=0, few=True, **kw):
    """Dense or grouped projection; see csrc/lib.py: gemm_simt for the keyword arguments.  `even_groups`: the groups' number,
    where all of them have equally many rows whatever the step (what `group_offsets` says too).  `few` False: a handful of tokens
    goes to the tcgen05 kernel all the same."""
    if use_tensor_cores and a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16:
        # products with many tokens go to the two-SM kernel, dense or grouped (it refuses, launching nothing, what it
        # does not take: few tokens per group, a row gather; features that are no multiple of 256 where they don't pay)
        rows, n = kw.get("m_rows", a.shape[0]), out.shape[1]
        # a handful of tokens: weights straight into registers (refuses, launching nothing, where the tcgen05 kernel is faster)
        if few and (even_groups or rows <= 32) and K.gemm_few(a, w, out, mode, even_groups=even_groups, **kw):
            return
        if use_paired_kernel and not single_cta_products.depth and "a_rows" not in kw and rows >= 512 and K.gemm_tc_pair(
                a, w, out, mode, any_features=bool(n % 256) and K.gemm_tc_pair_pays(rows, n, a.shape[1], mode in K.GATED_MODES), **kw):
            return
        if K.gemm_tc(a, w, out, mode, **kw):
            return
    K.gemm_simt(a, w, out, mode, **kw)
