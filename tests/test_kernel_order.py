"""An order that the kernels' sources have to keep, read from the sources: a kernel lets its successors start (programmatic
dependent launch) only when it has its tensor memory.  A successor that started earlier on the same SM could take the
columns and keep them until this kernel ends, which itself waits for them: neither would ever go on."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpi_b200", "csrc")
ALLOCATES = re.compile(r"tcgen05\.alloc|\btmem_alloc\(")


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\([^;{]*\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield f"{name}:{m.group(1)}", text[m.end():end]


KERNELS = dict(_kernels())
WITH_TENSOR_MEMORY = sorted(k for k, body in KERNELS.items() if ALLOCATES.search(body))


def test_the_kernels_with_tensor_memory_are_found():
    found = {k.split(":")[1] for k in WITH_TENSOR_MEMORY}
    assert {"gemm_tc_kernel", "gemm_tc_pair_kernel", "gemm_tc_pair_persistent_kernel", "attention_prefill_kernel",
            "latent_prefill_kernel"} <= found and len(KERNELS) > 60


@pytest.mark.parametrize("name", WITH_TENSOR_MEMORY)
def test_successors_start_after_the_tensor_memory_is_allocated(name):
    body = KERNELS[name]
    starts = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
    allocated = ALLOCATES.search(body).end()
    assert all(s > allocated and "__syncthreads" in body[allocated:s] for s in starts)


def test_a_pair_of_ctas_has_its_two_sms_to_itself():
    """The kernels on CTA pairs allocate tensor memory on two SMs at once.  Two pairs that shared an SM pair could wait for each
    other's half, so each of their launches takes more than half of an SM's 228 KB of shared memory."""
    text = open(os.path.join(CSRC, "gemm_tc_pair.cu")).read()
    alone = re.search(r"constexpr int kAlone = (\d+) \* 1024;", text)
    assert alone and 2 * int(alone.group(1)) > 228
    launches = re.findall(r"constexpr int SMEM = [^;]*;\s*(static_assert\(SMEM >= kAlone,)?", text)
    assert len(launches) == 3 and all(launches)
    pairs = [k for k, body in KERNELS.items() if "tcgen05.alloc.cta_group::2" in body]
    assert sorted(pairs) == ["gemm_tc_pair.cu:gemm_tc_pair_" + k for k in ("dual_kernel", "kernel", "persistent_kernel")]


def test_kernels_on_cta_pairs_are_not_started_early():
    """Launched behind row kernels of many blocks before those had ended, they did not always return."""
    text = open(os.path.join(CSRC, "gemm_tc_pair.cu")).read()
    assert text.count("cudaLaunchKernelEx(") == 2 and "cudaLaunchAttributeProgrammaticStreamSerialization" not in text
    assert "launch_pdl(" not in text


def test_kernels_that_allocate_through_a_helper_keep_the_order_too():
    """`tensor_begin` (recurrent_chunks.cu) allocates and meets; what calls it lets successors start after it."""
    text = open(os.path.join(CSRC, "recurrent_chunks.cu")).read()
    helper = text[text.index("void tensor_begin("):]
    helper = helper[:helper.index("\n}\n")]
    assert helper.index("tcgen05.alloc") < helper.index("__syncthreads()")
    users = {k: body for k, body in KERNELS.items() if "tensor_begin(" in body}
    assert {k.split(":")[1] for k in users} == {"chunk_state_kernel", "chunk_out_kernel", "chunk_out_step_kernel"}
    assert all(body.index("tensor_begin(") < body.index("pdl_launch_dependents()") for body in users.values())


def _before_the_wait(body):
    return body[:body.index("pdl_wait()")]


def test_index_arrays_are_read_before_the_wait_by_the_named_kernels_only():
    """They come from copies that end before a step's first kernel.  Anything else, cached rows above all, is written by kernels
    that may still be running when a kernel starts; `attention_decode` alone reads older pages early."""
    arrays = re.compile(r"\b(token_pos|token_seq|seq_slot|seq_tok0|seq_new|seq_start|page_table|tile_tok0|tile_rows)\s*\[")
    waiting = {k.split(":")[1]: _before_the_wait(body) for k, body in KERNELS.items() if "pdl_wait()" in body}
    assert {k for k, text in waiting.items() if arrays.search(text)} == {
        "attention_decode_kernel", "qkv_post_d128_kernel", "qkv_conv_rotate_kernel", "head_turn_kernel"}
    cached = re.compile(r"\bp\.(cache|k_cache|v_cache|q|state)\b|load_kv\(|load_tile\(")
    assert {k for k, text in waiting.items() if cached.search(text)} == {"attention_decode_kernel"}


@pytest.mark.parametrize("name", ["attention_decode.cu:attention_decode_kernel", "attention_prefill.cu:attention_prefill_kernel",
                                  "attention_simt.cu:attention_general_kernel", "attention_simt.cu:attention_f32_tile_kernel"])
def test_attention_over_cached_keys_waits_before_its_successors_start(name):
    """`attention_decode` of a later step reads rows of earlier positions before its own wait: they have been stored once the
    attention kernel behind their launch has waited, and whatever starts after it finds them."""
    body = KERNELS[name]
    starts = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
    assert all(body.index("pdl_wait()") < s for s in starts)


@pytest.mark.parametrize("name", ["chunk_state_kernel", "chunk_out_kernel", "chunk_out_step_kernel"])
def test_tiles_of_the_chunked_recurrences_end_with_one_decision(name):
    """A wait runs out for some threads and not for others.  In the loop over a block's tiles, which ends when one has, every
    barrier of the block is one that decides for all of them, so none meets another barrier than its neighbours."""
    body = KERNELS["recurrent_chunks.cu:" + name]
    start = body.index("for (int i = 0; i < count && ok; ++i) {")
    depth, end = 0, start
    while depth or "{" not in body[start:end]:
        depth += {"{": 1, "}": -1}.get(body[end], 0)
        end += 1
    loop = body[start:end]
    assert "mbar_wait(" in loop and "__syncthreads()" not in loop
    assert name == "chunk_state_kernel" or loop.rindex("ok = __syncthreads_and(ok) != 0;") > loop.rindex("mbar_wait(")
