"""The recurrences in chunks against a token-by-token scan in 64 bits, and against the float32 scan's own error."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _plain(a, k, q, v, S, beta=None):
    """S <- diag(a) S; S += k u^T with u = v, or beta (v - S^T k); o = S^T q.  a, k, q [T, H, N], v [T, H, Dv], S [H, N, Dv]."""
    S, o = S.clone(), torch.empty_like(v)
    for t in range(v.shape[0]):
        S *= a[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hnv,hn->hv", S, k[t]))
        S += k[t][:, :, None] * u[:, None, :]
        o[t] = torch.einsum("hnv,hn->hv", S, q[t])
    return o, S


def _batch(new, slots):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    tok0 = [sum(new[:i]) for i in range(len(new))]
    return SimpleNamespace(n_seqs=len(new), n_new=new, max_new=max(new), seq_slot=i32(slots), seq_tok0=i32(tok0), seq_new=i32(new))


# edges of a chunk of 64 (one token less and more, one token), unequal sequences, segments shorter than the step, heads that
# share q and k, decays from none to all, both sizes of a state's rows and one to four tiles of columns
@pytest.mark.parametrize("kind", ["rows", "step", "delta"])
@pytest.mark.parametrize("new,seg,rows,cols,decays", [
    ([64], 1, 64, 64, "slow"), ([65], 2, 128, 64, "fast"), ([63, 1, 130], 3, 64, 128, "slow"), ([300], 2, 128, 256, "mixed"),
    ([127, 128, 129], 1, 128, 128, "mixed"), ([1], 1, 64, 64, "none"), ([513, 70], 20, 64, 192, "fast"),
    ([2] * 40 + [200, 3], 5, 64, 64, "mixed")])
def test_chunks_equal_the_scan(kind, new, seg, rows, cols, decays):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV)
    T, H, hpg, B = sum(new), 4, 2, len(new)
    G = H // hpg
    k, q, v = randn(T, G * rows), randn(T, G * rows), randn(T, H * cols + 4)[:, :H * cols]
    if kind == "delta":                                      # unit keys, as the mixer's are
        k = torch.nn.functional.normalize(k.view(T, G, rows), dim=-1).view(T, G * rows)
    skip = None
    if kind == "step":
        raw, bias, a_log, skip = randn(T, H), randn(H), randn(H), randn(H)
        a_log += {"slow": -4.0, "fast": 2.0, "mixed": 0.0, "none": -40.0}[decays]
        kw = dict(dt=raw, dt_bias=bias, a_log=a_log, skip=skip)
        dt = torch.nn.functional.softplus(raw.double() + bias.double())
        a = torch.exp(-torch.exp(a_log.double()) * dt)[:, :, None].expand(T, H, rows)
    else:
        # z such that sigmoid(z + bias)^(1 / tau) covers the decays; -inf and inf give 0 and 1
        a = {"slow": 0.9 + 0.1 * rand(T, H, rows), "fast": rand(T, H, rows) ** 4, "none": torch.ones(T, H, rows, device=DEV),
             "mixed": (rand(T, H, rows) * 1.5).clamp(max=1.0) * (rand(T, H, rows) > 0.02)}[decays]
        kw = dict(z=torch.logit(a.double() ** 2).float().view(T, H * rows), z_bias=randn(H * rows), tau=2.0)
        zd = (kw["z"].double() + kw["z_bias"].double()).view(T, H, rows)
        a = torch.sigmoid(zd) ** 0.5
        if kind == "delta":                                  # its decays: exp(-rate softplus(z + bias))
            kw.update(beta=randn(T, H), decay_kind=1, a_log=randn(H), z=kw["z"].clamp(min=-30.0))
            zd = (kw["z"].double() + kw["z_bias"].double()).view(T, H, rows)
            a = torch.exp(-torch.exp(kw["a_log"].double())[:, None] * torch.nn.functional.softplus(zd))
    slots = [B - i for i in range(B)]                        # another order, slot 0 unused
    state = randn(B + 1, H, rows, cols)
    batch, q_scale = _batch(new, slots), 0.25
    per = K.linear_chunks_scratch(H, hpg, rows, cols, z=kw.get("z"), beta=kw.get("beta"))
    scratch = torch.full((seg * per,), float("nan"), device=DEV)             # nothing is read that was not written
    S, out = state.clone(), torch.full((T, H * cols), float("nan"), device=DEV)
    size = dict(n_heads=H, heads_per_group=hpg, n_rows=rows, n_cols=cols)
    K.linear_chunks(k, q, v, S, out, batch, scratch=scratch, q_scale=q_scale, **size, **kw)
    S2, out2 = state.clone(), torch.empty_like(out)
    K.linear_scan(k, q, v, S2, out2, batch, q_scale=q_scale, **size, **kw)
    assert torch.equal(S[0], state[0])
    kd, qd = (x.double().view(T, G, rows).repeat_interleave(hpg, 1) for x in (k, q))
    vd, t0 = v.double().reshape(T, H, cols), 0
    for n, slot in zip(new, slots):
        sl = slice(t0, t0 + n)
        vv = vd[sl] * (dt[sl][:, :, None] if kind == "step" else 1.0)
        beta = torch.sigmoid(kw["beta"].double()[sl]) if kind == "delta" else None
        o, ref = _plain(a.double()[sl], kd[sl], qd[sl] * q_scale, vv, state[slot].double(), beta)
        if skip is not None:
            o = o + skip.double()[:, None] * vd[sl]
        err = lambda x, y: float((x.double() - y).norm() / y.norm())
        # the scan's own error, and 2^-22 for sums of 64 terms taken in another order
        assert err(out[sl].view(n, H, cols), o) <= 1.5 * err(out2[sl].view(n, H, cols), o) + 2.0 ** -22
        assert err(S[slot], ref) <= 1.5 * err(S2[slot], ref) + 2.0 ** -22
        t0 += n


@pytest.mark.parametrize("kind", ["rows", "step", "delta"])
def test_an_output_reads_nothing_of_later_tokens(kind):
    """A NaN in a token's q, k, v and decay leaves the bits of every earlier token's output as they were."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(2)
    T, H, rows, cols, at = 150, 2, 64, 64, 83
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x = {n: randn(T, H * rows) * 0.2 for n in ("k", "q", "v")}
    fixed = {}
    if kind == "step":
        x.update(dt=randn(T, H))
        fixed = dict(dt_bias=randn(H), a_log=randn(H))
    else:
        x.update(z=torch.rand(T, H * rows, generator=g, device=DEV))
        if kind == "delta":
            x.update(beta=randn(T, H))
    got = []
    for broken in (False, True):
        y = {n: t.clone() for n, t in x.items()}
        if broken:
            for t in y.values():
                t[at] = float("nan")
        per = K.linear_chunks_scratch(H, 1, rows, cols, z=y.get("z"), beta=y.get("beta"))
        out = torch.zeros(T, H * cols, device=DEV)
        K.linear_chunks(y.pop("k"), y.pop("q"), y.pop("v"), torch.zeros(1, H, rows, cols, device=DEV), out, _batch([T], [0]),
                        scratch=torch.empty(3 * per, device=DEV), n_heads=H, heads_per_group=1, n_rows=rows,
                        n_cols=cols, **y, **fixed)
        got.append(out)
    assert torch.equal(got[0][:at], got[1][:at]) and bool(got[1][at:].isnan().all())


@pytest.mark.parametrize("kind", ["rows", "delta"])
def test_the_skip_adds_the_values_themselves(kind):
    """With row decays and with the delta rule, whose sums take corrected values: the scan's outputs with a skip."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(9)
    new, H, rows, cols = [70, 130], 2, 64, 128
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    T = sum(new)
    k, q, v = torch.nn.functional.normalize(randn(T, H, rows), dim=-1).view(T, -1), randn(T, H * rows), randn(T, H * cols)
    kw = dict(z=randn(T, H * rows), z_bias=randn(H * rows), skip=randn(H), n_heads=H, heads_per_group=1, n_rows=rows, n_cols=cols)
    if kind == "delta":
        kw.update(beta=randn(T, H), decay_kind=1, a_log=randn(H))
    per = K.linear_chunks_scratch(H, 1, rows, cols, z=kw["z"], beta=kw.get("beta"))
    outs, state = [], randn(2, H, rows, cols)
    for fn, extra in ((K.linear_scan, {}), (K.linear_chunks, dict(scratch=torch.empty(5 * per, device=DEV)))):
        S, out = state.clone(), torch.empty(T, H * cols, device=DEV)
        fn(k, q, v, S, out, _batch(new, [0, 1]), **kw, **extra)
        outs += [out, S]
    # float32 sums of up to 64 + 64 terms and of the states' rows in two orders
    for x, y in ((outs[0], outs[2]), (outs[1], outs[3])):
        assert float((x - y).norm() / x.norm()) <= 2.0 ** -18


# more tiles of columns than a block takes, counts that do not come out even, groups of an odd number of heads
@pytest.mark.parametrize("kind,H,hpg,rows,cols", [("step", 10, 5, 128, 64), ("step", 24, 12, 64, 128), ("rows", 10, 1, 64, 192),
                                                  ("rows", 3, 1, 128, 1024), ("delta", 6, 3, 128, 256), ("step", 9, 9, 128, 192)])
def test_blocks_of_several_tiles(kind, H, hpg, rows, cols):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(7)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    new, G = [1000, 37, 1300], H // hpg
    T = sum(new)
    k, q, v = torch.nn.functional.normalize(randn(T, G, rows), dim=-1).view(T, -1), randn(T, G * rows), randn(T, H * cols)
    kw = dict(n_heads=H, heads_per_group=hpg, n_rows=rows, n_cols=cols, q_scale=0.1)
    if kind == "step":
        kw.update(dt=randn(T, H), dt_bias=randn(H) - 3, a_log=randn(H), skip=randn(H))
    else:
        kw.update(z=randn(T, H * rows), z_bias=randn(H * rows), tau=16.0)
        if kind == "delta":
            kw.update(beta=randn(T, H), decay_kind=1, a_log=randn(H) - 3)
    per = K.linear_chunks_scratch(H, hpg, rows, cols, z=kw.get("z"), beta=kw.get("beta"))
    outs, state = [], randn(4, H, rows, cols)
    for fn, extra in ((K.linear_scan, {}), (K.linear_chunks, dict(scratch=torch.full((40 * per,), float("nan"), device=DEV)))):
        S, out = state.clone(), torch.zeros(T, H * cols, device=DEV)
        fn(k, q, v, S, out, _batch(new, [2, 0, 3]), **kw, **extra)
        outs.append((out, S))
    assert torch.equal(outs[1][1][1], state[1])
    for a, b in zip(*outs):
        # two float32 recurrences of 1,300 tokens, each some 2^-24 a token off (their errors against 64 bits are below 2e-6)
        assert float((a - b).norm() / a.norm()) < 1e-5 and bool(b.isfinite().all())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_values_that_are_no_numbers_reach_the_outputs_that_see_them(value):
    """One value of one column: the outputs of that column from its token on are no finite numbers, all others keep their bits."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(4)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    T, H, rows, cols, at = 130, 2, 64, 128, 70
    k, q, v, z = randn(T, H * rows), randn(T, H * rows), randn(T, H * cols), randn(T, H * rows)
    got = []
    for x in (0.5, value):
        v[at, cols + 3] = x
        per = K.linear_chunks_scratch(H, 1, rows, cols, z=z)
        out = torch.zeros(T, H * cols, device=DEV)
        K.linear_chunks(k, q, v, torch.zeros(1, H, rows, cols, device=DEV), out, _batch([T], [0]), scratch=torch.empty(3 * per, device=DEV),
                        n_heads=H, heads_per_group=1, n_rows=rows, n_cols=cols, z=z, tau=4.0)
        got.append(out)
    same = torch.ones(T, H * cols, dtype=torch.bool, device=DEV)
    same[at:, cols + 3] = False
    assert torch.equal(got[0][same], got[1][same]) and not bool(got[1][~same].isfinite().any())


# what no three bfloat16 terms hold: infinities, and numbers that bfloat16 rounds to one; tiles of 64 and of 128 columns, a tile
# that two heads share, and (with 16 groups) blocks of several tiles
@pytest.mark.parametrize("kind,groups,hpg,cols,segs", [
    ("rows", 2, 1, 64, 1), ("rows", 2, 1, 128, 1), ("rows", 2, 1, 192, 3), ("rows", 16, 1, 1024, 4), ("step", 2, 3, 64, 3), ("step", 2, 1, 128, 1),
    ("step", 2, 2, 192, 3), ("step", 16, 12, 64, 4), ("delta", 2, 1, 64, 3), ("delta", 2, 1, 128, 1), ("delta", 16, 1, 1024, 4)])
@pytest.mark.parametrize("what,value", [("v", float("inf")), ("v", float("-inf")), ("v", 3.4e38), ("v", -3.39e38), ("k", float("inf")),
                                        ("q", float("inf")), ("state", float("-inf")), ("state", 3.4e38)])
def test_numbers_without_bfloat16_terms(kind, groups, hpg, cols, segs, what, value):
    """One such number: outputs and states that do not see it keep their bits, the others are the scan's, infinities with its
    signs (but where an infinity meets one of its own column, as in all later tokens of the delta rule, and a query's, whose
    product with a state is taken in two parts: there no finite numbers)."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(6)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    G, rows, T, at, n = groups, 64, 200, 70, 5
    H = G * hpg
    h, col = hpg - 1 if hpg > 1 else 1, 3 if cols < 1024 else 700
    grp = h // hpg
    x = {"k": randn(T, G * rows).abs() * 0.05 + 0.01, "q": randn(T, G * rows).abs() * 0.05 + 0.01, "v": randn(T, H * cols)}
    state = randn(1, H, rows, cols)
    size = dict(n_heads=H, heads_per_group=hpg, n_rows=rows, n_cols=cols)
    if kind == "step":
        kw = dict(dt=randn(T, H), dt_bias=0.3 * randn(H) - 6, a_log=randn(H) - 2)      # (step sizes below one)
    else:
        kw = dict(z=randn(T, H * rows) + 2, z_bias=randn(H * rows), tau=4.0)
        if kind == "delta":
            kw.update(beta=randn(T, H), decay_kind=1, a_log=randn(H) - 3)
    per = K.linear_chunks_scratch(H, hpg, rows, cols, z=kw.get("z"), beta=kw.get("beta"))
    got = []
    for fn, broken in ((K.linear_chunks, False), (K.linear_chunks, True), (K.linear_scan, True)):
        y, S, out = {m: t.clone() for m, t in x.items()}, state.clone(), torch.zeros(T, H * cols, device=DEV)
        if broken:
            if what == "state":
                S[0, h, n, col] = value
            else:
                y[what][at, {"v": h * cols + col, "k": grp * rows + n, "q": grp * rows + n}[what]] = value
        extra = dict(scratch=torch.full((segs * per,), float("nan"), device=DEV)) if fn is K.linear_chunks else {}
        fn(y["k"], y["q"], y["v"], S, out, _batch([T], [0]), **size, **kw, **extra)
        got.append((out.view(T, H, cols), S[0]))
    sees, holds = torch.zeros(T, H, cols, dtype=torch.bool, device=DEV), torch.zeros(H, rows, cols, dtype=torch.bool, device=DEV)
    if what in ("v", "state"):
        sees[at if what == "v" else 0:, h, col] = holds[h, :, col] = True
    elif what == "k":
        sees[at:, grp * hpg:(grp + 1) * hpg] = holds[grp * hpg:(grp + 1) * hpg] = True
    else:
        sees[at, grp * hpg:(grp + 1) * hpg] = True
    (o0, s0), (o1, s1), (o2, s2) = got
    assert torch.equal(o0[~sees], o1[~sees]) and torch.equal(s0[~holds], s1[~holds])
    if value in (3.4e38, -3.39e38):
        assert bool(o1.isfinite().all()) and bool(s1.isfinite().all())
        # float32 sums of up to 128 terms and products of 200 decays, of numbers with no cancellation to speak of
        for a, b, m in ((o1, o2, sees), (s1, s2, holds)):
            assert float((a[m] / 3e38 - b[m] / 3e38).norm()) <= 2.0 ** -16 * float((b[m] / 3e38).norm())
        return
    if what == "q" or kind == "delta":
        assert not bool(o1[at][sees[at]].isfinite().any()) and torch.equal(o1.isfinite(), o2.isfinite())
        return
    if what == "v":
        o2[at, h, col] = o1[at, h, col]                      # (the scan adds the value times a skip of zero: NaN)
    for a, b in ((o1, o2), (s1, s2)):
        assert torch.equal(a.isposinf(), b.isposinf()) and torch.equal(a.isneginf(), b.isneginf()) and torch.equal(a.isnan(), b.isnan())
    assert bool(o1[sees].isinf().all())


# tiles of 128 columns over a group's heads: two heads side by side, a half tile at the end, heads of one and a half tiles
@pytest.mark.parametrize("hpg,cols,rows", [(1, 64, 64), (3, 64, 128), (3, 192, 64), (8, 64, 128), (2, 128, 64)])
def test_heads_that_share_a_tile_stay_apart(hpg, cols, rows):
    """One decay per head: against the scan in 64 bits, and with a head whose step sizes and values are no numbers the other
    heads' outputs and states keep their bits."""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(11)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    T, G = 150, 2
    H = G * hpg
    k, q, v, raw, bias, a_log, skip = randn(T, G * rows), randn(T, G * rows), randn(T, H * cols), randn(T, H), randn(H), randn(H), randn(H)
    state = randn(1, H, rows, cols)
    size = dict(n_heads=H, heads_per_group=hpg, n_rows=rows, n_cols=cols)
    got = []
    for broken in (False, True):
        r, w = raw.clone(), v.clone()
        if broken:
            r[40:, hpg - 1], w[70, (hpg - 1) * cols:hpg * cols] = float("nan"), float("inf")
        S, out = state.clone(), torch.full((T, H * cols), float("nan"), device=DEV)
        per = K.linear_chunks_scratch(H, hpg, rows, cols)
        K.linear_chunks(k, q, w, S, out, _batch([T], [0]), scratch=torch.empty(2 * per, device=DEV), q_scale=0.25, dt=r, dt_bias=bias,
                        a_log=a_log, skip=skip, **size)
        got.append((out.view(T, H, cols), S[0]))
    others = [h for h in range(H) if h != hpg - 1]
    assert torch.equal(got[0][0][:, others], got[1][0][:, others]) and torch.equal(got[0][1][others], got[1][1][others])
    assert torch.equal(got[0][0][:40], got[1][0][:40]) and bool(got[1][0][40:, hpg - 1].isnan().all())
    S2, out2 = state.clone(), torch.empty(T, H * cols, device=DEV)
    K.linear_scan(k, q, v, S2, out2, _batch([T], [0]), q_scale=0.25, dt=raw, dt_bias=bias, a_log=a_log, skip=skip, **size)
    dt = torch.nn.functional.softplus(raw.double() + bias.double())
    a = torch.exp(-torch.exp(a_log.double()) * dt)[:, :, None].expand(T, H, rows)
    kd, qd = (x.double().view(T, G, rows).repeat_interleave(hpg, 1) for x in (k, q))
    vd = v.double().view(T, H, cols)
    o, ref = _plain(a, kd, qd * 0.25, vd * dt[:, :, None], state[0].double())
    o = o + skip.double()[:, None] * vd
    err = lambda x, y: float((x.double() - y).norm() / y.norm())
    # the scan's own error, and 2^-22 for sums of 64 terms taken in another order
    assert err(got[0][0], o) <= 1.5 * err(out2.view(T, H, cols), o) + 2.0 ** -22
    assert err(got[0][1], ref) <= 1.5 * err(S2[0], ref) + 2.0 ** -22


@pytest.mark.parametrize("kind", ["rows", "step"])
def test_sums_lean_to_neither_side(kind):
    """States and outputs of one chunk without decays are plain sums of products.  Against 64 bits their mean error in the direction
    of the sum stays below 2^-26 of the mean sum: the tensor core truncates, 2^-25 of a sum and more if nothing is given back,
    float32 rounding to nearest none.  (65,536 sums and more, each some 2^-24 off: their mean is known to 2^-32.)"""
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(8)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    T, H, rows, cols = 64, 8, 128, 128
    k, q, v = randn(T, H * rows), randn(T, H * rows), randn(T, H * cols)
    kw = dict(dt=torch.zeros(T, H, device=DEV), dt_bias=torch.zeros(H, device=DEV), a_log=torch.full((H,), -60.0, device=DEV)) if kind == "step" \
        else dict(z=torch.full((T, H * rows), float("inf"), device=DEV))
    per = K.linear_chunks_scratch(H, 1, rows, cols, z=kw.get("z"))
    S, out = torch.zeros(1, H, rows, cols, device=DEV), torch.zeros(T, H * cols, device=DEV)
    K.linear_chunks(k, q, v, S, out, _batch([T], [0]), scratch=torch.zeros(per, device=DEV), n_heads=H, heads_per_group=1, n_rows=rows,
                    n_cols=cols, **kw)
    kd, qd, vd = (x.double().view(T, H, -1) for x in (k, q, v))
    if kind == "step":
        vd = vd * float(torch.nn.functional.softplus(torch.zeros(1, device=DEV)))            # (the step size as float32 has it)
    o, ref = _plain(torch.ones(T, H, rows, device=DEV, dtype=torch.float64), kd, qd, vd, S[0].double() * 0)
    lean = lambda x, y: abs(float(((x.double() - y) * y.sign()).mean() / y.abs().mean()))
    assert lean(S[0], ref) <= 2.0 ** -26 and lean(out.view(T, H, cols), o) <= 2.0 ** -26
