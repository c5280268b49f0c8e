"""Prompt attention over a cached latent with formed keys and values: its kernels against 64-bit arithmetic on the same
operands, and the mixer's two forms against each other."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(starts, new, extra=2):
    """A batch, and pages for it in a scattered order: (batch, page table, number of pages)."""
    from cpi_b200.engine.batch import BatchStager
    blocks = [-(-(s + n) // 64) for s, n in zip(starts, new)]
    order = torch.randperm(sum(blocks) + extra, generator=torch.Generator().manual_seed(1)).int()
    table = torch.zeros(len(new), max(blocks), dtype=torch.int32)
    at = 0
    for i, b in enumerate(blocks):
        table[i, :b] = order[at:at + b]
        at += b
    stager = BatchStager(DEV)
    batch = stager.stage(list(range(len(new))), starts, [[0] * n for n in new], [[] for _ in new], torch.bfloat16)
    batch.keep = stager
    return batch, table.to(DEV), len(order)


# edges: one row, a tile less / more than 128 and 256 queries, key tiles that end inside and at a page, a prompt that goes
# on behind cached positions, windows smaller and larger than a tile, several sequences, more heads than one group
@pytest.mark.parametrize("starts,new,window,sink,heads", [
    ([0], [2], 0, False, 1), ([0], [128], 0, False, 3), ([0], [129], 0, True, 2), ([0], [257], 0, False, 2),
    ([0, 0, 0], [63, 300, 64], 0, True, 2), ([333], [54], 0, False, 4), ([100, 0, 700], [200, 31, 513], 0, False, 3),
    ([0], [700], 1, False, 1), ([0], [600], 100, True, 2), ([517, 0], [400, 150], 300, False, 2), ([0], [1025], 4096, False, 1)])
def test_latent_prefill_kernels(starts, new, window, sink, heads):
    from cpi_b200.csrc import lib as K
    batch, table, n_pages = _step(starts, new)
    g = torch.Generator(device=DEV).manual_seed(7)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    rank, T, H, scale = 72, sum(new), heads + 1, 0.1           # the launch takes the heads 1 .. of H
    pages = randn(n_pages, 1, 64, rank + 64).bfloat16()
    end = starts[0] + new[0] - 1
    pages[table[0, end // 64].item(), 0, end % 64 + 1:] = float("nan")               # stale contents behind a sequence's end
    first = [K.latent_first_row(s, window) for s in starts]
    R = sum(s + n - f for s, n, f in zip(starts, new, first))
    rows = torch.full((R, rank + 64), float("nan"), device=DEV).bfloat16()
    K.latent_key_rows(pages, rows, table, batch, window=window)
    want = torch.cat([pages[table[i].long()].reshape(-1, rank + 64)[f:s + n] for i, (s, n, f) in enumerate(zip(starts, new, first))])
    assert torch.equal(rows, want)
    q, kv = randn(T, H * 192).bfloat16(), randn(R, heads * 256).bfloat16()
    sinks = randn(H) if sink else None
    out = torch.zeros(T, H * 128, device=DEV, dtype=torch.bfloat16)
    K.latent_prefill(q, kv, rows, out, batch, heads=(1, H), out_heads=H, rank=rank, scale=scale, sink=sinks, window=window)
    torch.cuda.synchronize()
    assert int(K.tc_error_flag(DEV)) == 0 and not out[:, :128].any()
    if len(new) > 1:                     # nothing of the second sequence reaches the first one's rows
        broken, again = kv.clone(), torch.zeros_like(out)
        broken[starts[0] + new[0] - first[0]:] = float("nan")
        K.latent_prefill(q, broken, rows, again, batch, heads=(1, H), out_heads=H, rank=rank, scale=scale, sink=sinks, window=window)
        assert torch.equal(again[:new[0]], out[:new[0]])
    t0 = r0 = 0
    for s, n, f in zip(starts, new, first):
        m = s + n - f
        dist = torch.arange(s, s + n, device=DEV)[:, None] - torch.arange(f, s + n, device=DEV)[None, :]
        hide = (dist < 0) | (dist >= (window or 1 << 30))
        for h in range(heads):
            k = torch.cat([kv[r0:r0 + m, h * 256:h * 256 + 128], rows[r0:r0 + m, rank:]], 1).double()
            v = kv[r0:r0 + m, h * 256 + 128:(h + 1) * 256].double()
            x = (q[t0:t0 + n, (h + 1) * 192:(h + 2) * 192].double() @ k.T * scale).masked_fill(hide, -math.inf)
            if sink:
                x = torch.cat([x, sinks[h + 1].double().expand(n, 1)], 1)
            ref = torch.softmax(x, 1)[:, :m] @ v
            # every probability is rounded to bfloat16's 8 significant bits (by 2^-8 of it at most), the output once more
            bound = 2.0 ** -8 * (float(v.abs().max()) + ref.abs()) * 1.05
            assert bool(((out[t0:t0 + n, (h + 1) * 128:(h + 2) * 128].double() - ref).abs() <= bound).all())
        t0, r0 = t0 + n, r0 + m


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("dim,rot,heads", [(128, 64, 3), (4, 8, 1), (100, 16, 5)])
def test_query_rows_are_rounded_after_their_rotation(dim, rot, heads, interleaved):
    from cpi_b200.csrc import lib as K
    g = torch.Generator(device=DEV).manual_seed(3)
    T = 37
    q = torch.randn(T, heads * (dim + rot) + 4, generator=g, device=DEV)[:, :heads * (dim + rot)]
    pos = torch.arange(5, 5 + T, device=DEV, dtype=torch.int32)
    freq = (1e4 ** (-torch.arange(rot // 2, device=DEV) * 2.0 / rot)).float()
    out = torch.empty(T, heads * (dim + rot), device=DEV, dtype=torch.bfloat16)
    K.latent_q_rows(q, freq, interleaved, out, pos, n_heads=heads, dim=dim, rot=rot, amplitude=1.25)
    x = q.double().view(T, heads, dim + rot)
    a = (pos.float()[:, None] * freq).double()[:, None]
    c, s = 1.25 * torch.cos(a), 1.25 * torch.sin(a)
    r = x[..., dim:]
    u, v = (r[..., 0::2], r[..., 1::2]) if interleaved else (r[..., :rot // 2], r[..., rot // 2:])
    y = (u * c - v * s, v * c + u * s)
    y = torch.stack(y, -1).flatten(-2) if interleaved else torch.cat(y, -1)
    want = torch.cat([x[..., :dim], y], -1).view(T, -1)
    # one rounding to 8 significant bits (2^-8 of the value at most), the float32 rotation before it at most 2^-21 of the
    # row's largest element
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() * 1.01 + 2.0 ** -21 * q.abs().max()).all())


@pytest.mark.parametrize("starts,new,window,gate", [([0], [300], None, False), ([0, 200], [150, 90], None, True),
                                                    ([0, 0], [700, 64], 128, False)])
def test_both_forms_of_the_mixer_agree(starts, new, window, gate, monkeypatch):
    from cpi_b200.cache import CacheManager
    from cpi_b200.config.spec import PartSpec
    from cpi_b200.parts import CacheView, Workspace, build_part, latent
    from cpi_b200.weights import DictSource
    from cpi_b200.engine.batch import BatchStager
    rope = PartSpec("rope", {"head_dim": 64, "theta": 1e4, "pairing": "interleaved", "scaling": None})
    spec = PartSpec("latent_attention", {"hidden_size": 256, "heads": 3, "head_dim": 128, "rot_dim": 64, "value_dim": 128, "q_rank": 96,
                                         "kv_rank": 128, "softmax_scale": 192 ** -0.5, "norm_eps": 1e-6, "position": rope, "sink": True,
                                         "output_gate": gate, "window": None if window is None else {"kind": "sliding", "size": window}})
    mixer = build_part("mixer", spec, "", workspace=Workspace(DEV))
    g = torch.Generator(device=DEV).manual_seed(11)
    w = {r.name: ((0.05 * torch.randn(r.shape, generator=g, device=DEV)) + (1.0 if "ones" in r.init else 0.0)).bfloat16()
         for r in mixer.requirements()}
    mixer.load(DictSource(w), DEV)
    cache = CacheManager({0: mixer.kv_requirement()}, {}, max_tokens=2048, max_seqs=len(new), dtype=torch.bfloat16, device=DEV)
    slots = [cache.acquire() for _ in new]
    stager, got = BatchStager(DEV), {}
    past = [i for i, s in enumerate(starts) if s]
    h0 = torch.randn(sum(starts), 256, generator=g, device=DEV).bfloat16()
    if past:
        cache.prepare_step([slots[i] for i in past], [starts[i] for i in past])
        b = stager.stage([slots[i] for i in past], [0] * len(past), [[0] * starts[i] for i in past], [[]] * len(past), torch.bfloat16)
        mixer.forward(h0, torch.zeros(h0.shape, device=DEV), b, CacheView(cache, 0))
        cache.commit_step([slots[i] for i in past], [starts[i] for i in past])
    cache.prepare_step(slots, new)
    batch = stager.stage(slots, starts, [[0] * n for n in new], [[]] * len(new), torch.bfloat16)
    h = torch.randn(sum(new), 256, generator=g, device=DEV).bfloat16()
    for form in (True, False):
        monkeypatch.setattr(latent, "use_formed_keys", form)
        # groups of one head and of all heads at a time give the same bits
        for limit in ((1, 1 << 29) if form else (1,)):
            monkeypatch.setattr(latent, "FORMED_BYTES", limit)
            assert mixer._forms_keys(batch, torch.bfloat16, 64) is form
            out = torch.zeros(h.shape, device=DEV)
            mixer.forward(h, out, batch, CacheView(cache, 0))
            assert not form or form not in got or torch.equal(got[form], out)
            got[form] = out
    assert float((got[True] - got[False]).norm() / got[False].norm()) <= 1e-2      # two orders of bfloat16 roundings


def test_many_short_continuations_stay_with_the_cached_rows():
    from types import SimpleNamespace
    from cpi_b200.parts import latent

    def forms(starts, new, window=0, heads=16):
        m = SimpleNamespace(w_kv=0, d=128, r=64, dv=128, kv_rank=512, window=window, nh=heads)
        b = SimpleNamespace(is_decode=False, n_q_tiles=1, starts=starts, n_new=new)
        return latent.LatentAttentionMixer._forms_keys(m, b, torch.bfloat16, 64)
    assert forms([0], [2048]) and forms([0] * 40, [100] * 40) and forms([2000], [2]) and forms([100000], [512], 1024)
    assert not forms([1000] * 16, [2] * 16) and not forms([0] * 40, [20] * 40)


def test_a_prompt_without_room_for_keys_and_values_stays_with_the_cached_rows(monkeypatch):
    """The same bits as with the formed keys switched off, and nothing is written before the room is known."""
    from cpi_b200.cache import CacheManager
    from cpi_b200.config.spec import PartSpec
    from cpi_b200.csrc import lib as K
    from cpi_b200.parts import CacheView, Workspace, build_part, latent
    from cpi_b200.weights import DictSource
    from cpi_b200.engine.batch import BatchStager
    rope = PartSpec("rope", {"head_dim": 64, "theta": 1e4, "pairing": "interleaved", "scaling": None})
    spec = PartSpec("latent_attention", {"hidden_size": 256, "heads": 3, "head_dim": 128, "rot_dim": 64, "value_dim": 128, "q_rank": 96,
                                         "kv_rank": 128, "softmax_scale": 192 ** -0.5, "norm_eps": 1e-6, "position": rope, "sink": False})
    ws = Workspace(DEV)
    mixer = build_part("mixer", spec, "", workspace=ws)
    g = torch.Generator(device=DEV).manual_seed(11)
    w = {r.name: ((0.05 * torch.randn(r.shape, generator=g, device=DEV)) + (1.0 if "ones" in r.init else 0.0)).bfloat16()
         for r in mixer.requirements()}
    mixer.load(DictSource(w), DEV)
    cache = CacheManager({0: mixer.kv_requirement()}, {}, max_tokens=512, max_seqs=1, dtype=torch.bfloat16, device=DEV)
    slots = [cache.acquire()]
    cache.prepare_step(slots, [300])
    stager = BatchStager(DEV)
    batch = stager.stage(slots, [0], [[0] * 300], [[]], torch.bfloat16)
    h = torch.randn(300, 256, generator=g, device=DEV).bfloat16()

    def run():
        out = torch.zeros(h.shape, device=DEV)
        mixer.forward(h, out, batch, CacheView(cache, 0))
        return out
    run()
    monkeypatch.setattr(latent, "use_formed_keys", False)
    want = run()
    grown = ws.generation
    monkeypatch.setattr(latent, "use_formed_keys", True)
    for which in (0, 1):                                     # no room for the rows, or for the keys and values
        asked = []
        scratch = Workspace.scratch
        monkeypatch.setattr(Workspace, "scratch", lambda self, n, dt: asked.append(n) or (None if len(asked) == which + 1 else scratch(self, n, dt)))
        monkeypatch.setattr(K, "latent_key_rows", None)
        assert torch.equal(run(), want) and len(asked) == 2
        monkeypatch.setattr(Workspace, "scratch", scratch)
    # a longer context moves no buffer that a captured decode graph holds
    cache.commit_step(slots, [300])
    cache.prepare_step(slots, [200])
    batch = stager.stage(slots, [300], [[0] * 200], [[]], torch.bfloat16)
    h = h[:200]
    monkeypatch.undo()
    run()
    assert ws.generation == grown
