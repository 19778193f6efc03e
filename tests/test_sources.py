"""Rules that the CUDA sources keep, read from the sources themselves (no GPU)."""
from __future__ import annotations

import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pico-engine_b200", "csrc")


@pytest.mark.parametrize("name", ["linear_simt", "linear_fused", "linear_batch", "gemm_splitk", "attention_decode", "attention_diff"])
def test_cluster_barriers_are_of_the_form_that_lanes_may_reach_apart(name):
    """The kernels that merge ranges over a cluster come to its barrier from loops that the lanes of a warp leave at different times;
    the .aligned form is only defined where they arrive together."""
    with open(os.path.join(CSRC, name + ".cu")) as f:
        lines = [line for line in f if "barrier.cluster" in line]
    assert lines and not any(".aligned" in line for line in lines)


def test_float32_products_leave_their_cluster_together():
    """Up to 64 rows, the CTAs of linear_split.cu write sums into each other's shared memory, so none may end before all have sent, not even
    one whose waits ran out: no way out of the kernel but its end, a cluster barrier between the last sum sent and that end in
    every form, and a wait for the others' sums that the CTA's own give-up flag does not cut short."""
    with open(os.path.join(CSRC, "linear_split.cu")) as f:
        text = f.read()
    body = text[text.index("linear_split_kernel(const __grid_constant__"):text.index("static int sp_map")]
    behind = body[body.index("st.async"):]
    assert "return;" not in body
    arrive, finish = behind.index("barrier.cluster.arrive"), behind.index("sp_finish(")
    assert arrive < finish < behind.index("barrier.cluster.wait")
    assert not any("(sent" in line and "abort" in line for line in body.splitlines())


def test_streamed_decode_products_write_nothing_of_a_group_that_did_not_come():
    """A wait of linear_stream.cuh that runs out is told to the whole block before the group's results are written, and ends its loop over
    groups."""
    with open(os.path.join(CSRC, "linear_stream.cuh")) as f:
        text = f.read()
    body = text[text.index("linear_stream_kernel("):text.index("static int ls_launch_nt")]
    waits, told, writes = body.index("lf_bar_wait(bar"), body.index("__syncthreads_or("), body.index("p.out")
    assert waits < told < writes and "break;" in body[told:writes]
    assert body[waits:told].count("break;") == 1 and "late = true" in body[waits:told]


@pytest.mark.parametrize("name", ["prefill", "diff", "headmix", "latent"])
def test_prompt_kernels_read_nothing_before_the_kernel_in_front_has_ended(name):
    """The step's runs and the page table are inputs like any other: a kernel in front may be writing them."""
    with open(os.path.join(CSRC, f"attention_{name}_tcgen05.cu")) as f:
        body = f.read().split("__global__", 1)[1]
    assert body.index("pdl_wait();") < min(body.index(what) for what in ("p.tiles[", "p.block_table", "table["))


@pytest.mark.parametrize("name,kernel", [("linear_attention_tcgen05", "lm_prepare_kernel"), ("linear_attention_tcgen05", "lm_channels_kernel"), ("state_space_tcgen05", "sm_steps_kernel")])
def test_words_that_a_block_lowers_stand_before_any_thread_does(name, kernel):
    """One thread sets the words that tell of entries which are no numbers; the block meets before any other may change them, or its store
    could come behind theirs and forget a token."""
    with open(os.path.join(CSRC, name + ".cu")) as f:
        body = f.read().split(kernel + "(", 1)[1].split("__global__", 1)[0]
    body = body[body.index("seen = 0;"):]
    first = min(body.index(what) for what in ("lm_values(", "lm_put_mended(", "cm_report(", "cm_mend(", "atomicMin(") if what in body)
    assert "__syncthreads();" in body[:first]
