"""The recurrent mixers as a model runs them: the routes that their sizes and steps choose, against plain 64-bit mixers."""
import pytest
import torch

import plain_savenex
import plain_veredra

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mixer(kind, params, seed, dtype=torch.bfloat16):
    """(mixer, its weights by the mixer's names)."""
    from cpi_b200.config.spec import PartSpec
    from cpi_b200.parts import Workspace, build_part
    from cpi_b200.weights import DictSource
    mixer = build_part("mixer", PartSpec(kind, params), "", workspace=Workspace(DEV))
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = {}
    for r in mixer.requirements():
        t = torch.randn(r.shape, generator=g, device=DEV) * (0.3 if "conv" in r.name else 0.05)
        w[r.name] = (t + (1.0 if "ones" in r.init else 0.0)).to(dtype)
    mixer.load(DictSource(w), DEV)
    return mixer, {k: w[name].double().cpu() for k, name in mixer.tn.items()}


def _cache(mixer, n, dtype=torch.bfloat16):
    from cpi_b200.cache import CacheManager
    cache = CacheManager({}, {0: mixer.state_requirements()}, max_tokens=4096, max_seqs=n, dtype=dtype, device=DEV)
    return cache, [cache.acquire() for _ in range(n)]


def _step(mixer, cache, slots, starts, h, new):
    from cpi_b200.engine.batch import BatchStager
    from cpi_b200.parts import CacheView
    stager = BatchStager(DEV)
    cache.prepare_step(slots, new)
    batch = stager.stage(slots, starts, [[0] * n for n in new], [[] for _ in new], h.dtype)
    out = torch.zeros(h.shape, device=DEV)
    mixer.forward(h, out, batch, CacheView(cache, 0))
    cache.commit_step(slots, new)
    torch.cuda.synchronize()
    return out


GLA_NAMES = {"q": "q", "k": "k", "v": "v", "g": "g", "a1": "a1", "a2": "a2", "a2.b": "a2_bias", "norm": "norm", "o": "o"}


# decays whose first projection is part of the input product, the widest such, one more, and one that is no multiple of 8
@pytest.mark.parametrize("rank,rides", [(16, True), (64, True), (72, False), (128, False), (100, False)])
@pytest.mark.parametrize("T", [1, 40, 530])
def test_decays_of_a_wide_rank_take_the_tensor_cores(rank, rides, T, monkeypatch):
    from cpi_b200.csrc import lib as K
    m = {"heads": 2, "dim": 64, "vdim": 64, "tau": 16.0}
    mixer, w = _mixer("gla", {"hidden_size": 256, "heads": 2, "key_dim": 64, "value_dim": 64, "tau": 16.0, "decay_rank": rank,
                              "norm_eps": 1e-5}, rank)
    cache, slots = _cache(mixer, 1)
    h = torch.randn(T, 256, generator=torch.Generator(device=DEV).manual_seed(T), device=DEV).bfloat16()
    calls, simt = [], K.gemm_simt
    monkeypatch.setattr(K, "gemm_simt", lambda *a, **kw: calls.append(1) or simt(*a, **kw))
    out = _step(mixer, cache, slots, [0], h, [T])
    assert mixer.rides == rides and len(calls) == int(rides or rank % 8 != 0)      # (rows off 16 bytes are refused there)
    want = plain_veredra.gla_mixer(h.double().cpu(), m, lambda n: w[GLA_NAMES[n]], 1e-5)
    # bfloat16 rounds the gated heads before W_o (and a wide rank's rows): 2^-9 of each on average
    assert float((out.double().cpu() - want).norm() / want.norm()) <= 2.0 ** -8


def test_a_prompt_without_room_for_chunks_is_scanned(monkeypatch):
    from cpi_b200.csrc import lib as K
    from cpi_b200.parts import Workspace
    params = {"hidden_size": 256, "heads": 2, "key_dim": 64, "value_dim": 64, "tau": 16.0, "decay_rank": 16, "norm_eps": 1e-5}
    h = torch.randn(300, 256, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).bfloat16()
    outs = []
    for room in (True, False):
        mixer, _ = _mixer("gla", params, 5)
        cache, slots = _cache(mixer, 1)
        if not room:
            monkeypatch.setattr(Workspace, "scratch", lambda *a: None)
            monkeypatch.setattr(K, "linear_chunks", None)
        outs.append((_step(mixer, cache, slots, [0], h, [300]), cache.state_view(0, "s").clone()))
    for x, y in zip(*outs):                                  # two orders of float32 sums, bfloat16 rows into W_o
        assert float((x - y).norm() / y.norm()) <= 2.0 ** -8


MAMBA_NAMES = {"in": "in", "conv": "conv", "conv.b": "conv_bias", "dt_bias": "dt_bias", "A_log": "A_log", "D": "D", "norm": "norm", "o": "o"}
DELTA_NAMES = {"q": "q", "k": "k", "v": "v", "q.conv": "q_conv", "k.conv": "k_conv", "v.conv": "v_conv", "b": "b", "a1": "a1", "a2": "a2",
               "dt_bias": "dt_bias", "A_log": "A_log", "norm": "norm", "g1": "g1", "g2": "g2", "o": "o"}
KINDS = {
    "gla": ("gla", {"hidden_size": 192, "heads": 2, "key_dim": 64, "value_dim": 128, "tau": 16.0, "decay_rank": 16, "norm_eps": 1e-5},
            lambda h, w: plain_veredra.gla_mixer(h, {"heads": 2, "dim": 64, "vdim": 128, "tau": 16.0}, lambda n: w[GLA_NAMES[n]], 1e-5)),
    "mamba2": ("mamba2", {"hidden_size": 192, "heads": 4, "head_dim": 64, "state": 128, "groups": 2, "conv": 4, "norm_groups": 2,
                          "norm_eps": 1e-5},
               lambda h, w: plain_veredra.mamba2_mixer(h, {"heads": 4, "vdim": 64, "state": 128, "groups": 2, "norm_groups": 2},
                                                       lambda n: w[MAMBA_NAMES[n]], 1e-5)),
    "delta": ("gated_delta", {"hidden_size": 192, "heads": 2, "kv_heads": 1, "key_dim": 64, "value_dim": 64, "conv": 4, "decay_rank": 16,
                              "gate_rank": 16, "norm_eps": 1e-5},
              lambda h, w: plain_savenex.right_mixer(h, {n: w[m] for n, m in DELTA_NAMES.items()}, "",
                                                     {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64}, 1e-5)),
}


# a longest portion one short of the line, on it, and well past it beside short ones, with the chunks in one and in several segments; then
# a piece that goes on, and single tokens on the states that the prompt left
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("past,segments", [(-1, False), (0, False), (70, False), (70, True)])
def test_mixers_take_chunks_from_their_line_on(kind, past, segments, monkeypatch):
    from cpi_b200.csrc import lib as K
    from cpi_b200.parts import recurrent
    name, params, plain = KINDS[kind]
    line = recurrent.DELTA_CHUNKS_FROM if kind == "delta" else recurrent.CHUNKS_FROM
    new, more = [20, line + past, 65], [line, 3, 40]
    g = torch.Generator(device=DEV).manual_seed(past + 2)
    hs = [torch.randn(n + m + 2, 192, generator=g, device=DEV).bfloat16() for n, m in zip(new, more)]
    calls, chunks = [], K.linear_chunks

    def counted(*a, scratch, **kw):
        per = K.linear_chunks_scratch(kw["n_heads"], kw["heads_per_group"], kw["n_rows"], kw["n_cols"], z=kw["z"], beta=kw.get("beta"))
        calls.append(scratch.numel() // per)
        return chunks(*a, scratch=scratch, **kw)
    monkeypatch.setattr(K, "linear_chunks", counted)
    outs = {}
    for chunked in (True, False):
        monkeypatch.setattr(recurrent, "use_chunked_kernel", chunked)
        if segments:
            monkeypatch.setattr(recurrent, "CHUNK_BYTES", 1)
        mixer, w = _mixer(name, params, 3)
        cache, slots = _cache(mixer, 3)
        got, at = [[] for _ in new], [0, 0, 0]
        calls.clear()
        for step in (new, more, [1, 1, 1], [1, 1, 1]):
            rows = torch.cat([h[a:a + n] for h, a, n in zip(hs, at, step)])
            for i, y in enumerate(_step(mixer, cache, slots, list(at), rows, step).split(step)):
                got[i].append(y)
            at = [a + n for a, n in zip(at, step)]
        outs[chunked] = [torch.cat(x) for x in got]
        assert len(calls) == (0 if not chunked else 1 if past < 0 else 2)      # the second step's longest is on the line
        assert all(n == 1 if segments else n > 1 for n in calls)
    for i, h in enumerate(hs):
        want = plain(h.double().cpu(), w)
        err = [float((outs[c][i].double().cpu() - want).norm() / want.norm()) for c in (True, False)]
        # bfloat16 rows into W_o (and their activations): 2^-9 of each on average; the chunks no further off than the scan
        assert err[1] <= 2.0 ** -7 and err[0] <= 1.02 * err[1] + 2.0 ** -14
