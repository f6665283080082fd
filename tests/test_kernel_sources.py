"""Orders in the kernels' sources that no run can show to be wrong without hanging a GPU."""
import os
import re

from conftest import cg

CSRC = os.path.join(os.path.dirname(cg.__file__), "csrc")


def kernel(file, name):
    """The source of one kernel's definition."""
    text = open(os.path.join(CSRC, file)).read()
    begin = re.search(rf"\b{name}\(const __grid_constant__", text).start()
    return text[begin:text.index("\n}\n", begin)]


def places(body, *instructions):
    """Where each stands; all must stand there exactly once."""
    assert all(body.count(i) == 1 for i in instructions), [body.count(i) for i in instructions]
    return [body.index(i) for i in instructions]


def test_prompt_attention_takes_tmem_between_its_dependency_and_its_trigger():
    """A CTA that wants most of an SM's TMEM: after the wait no earlier kernel holds columns, and before the trigger no later
    kernel runs.  The other way round a dependent's CTA could hold columns and wait for a kernel that waits for them."""
    for name in ("k_attn_fa", "k_attn_fq"):
        wait, alloc, trigger = places(kernel("attention_fa.cu", name), "griddepcontrol.wait;", "tcgen05.alloc.", "griddepcontrol.launch_dependents;")
        assert wait < alloc < trigger


def test_pushes_to_a_cta_that_gave_up_are_counted_out_before_it_leaves():
    """A CTA of the decode GEMM that has given up on a wait may still be pushed to when every peer has passed the last cluster
    barrier (issued is not arrived).  It polls for the bytes whatever has been reported: a wait that ends early because the
    error is known would let it leave."""
    body = kernel("gemm_dec.cu", "k_gemm_dec")
    last = body.rindex("barrier.cluster.wait.acquire.aligned")
    assert "if (*cta_abort) mbar_drain(bar_x, 0, p.err);" in body[last:] and "mbar_wait" not in body[last:]
    common = open(os.path.join(CSRC, "tc_common.cuh")).read()
    drain = common[common.index("void mbar_drain("):]
    drain = drain[:drain.index("\n}\n")]
    assert "abort" not in drain and "DEV_TIMEOUT" not in drain and "limit" in drain


def test_the_step_counter_is_released_to_early_readers():
    """k_recur_decode reads its state before its dependency wait and trusts it if the step counter (ld.acquire) has not moved:
    whoever raises the counter has to release what the step wrote."""
    early = open(os.path.join(CSRC, "recurrent.cu")).read()
    assert early.count("ld.acquire.gpu.global.s64") == 2
    text = open(os.path.join(CSRC, "fused.cu")).read()
    assert "*pos_dev +=" not in text and "++*pos_dev" not in text
    raised = text[text.index("void step_done("):]
    assert "st.release.gpu.global.s64" in raised[:raised.index("\n}\n")]
    for name in ("k_argmax_finish", "k_argmax_finish_tp"):
        body = text[text.index(f" {name}("):]
        body = body[:body.index("\n}\n")]
        assert body.index("griddepcontrol.wait;") < body.index("step_done(pos_dev);")


def test_tiles_asked_for_with_a_stale_position_are_waited_for():
    """The decode attention asks for its first tiles with a position that may be a step old, and asks again where it was.  The
    first copies are waited for by a wait that reports when it gives up; after that the warp takes no tile.  A poll that
    says nothing would leave the barrier a phase behind, and the next wait would pass before its tile is there."""
    text = open(os.path.join(CSRC, "attn_decode.cuh")).read()
    item = text[text.index("void attn_dec_item("):]
    init = item.index("tc::mbar_init(bar_v, 1);")
    assert init < item.index("__syncwarp();\n    if (tid == 0) *cta_abort = 0;") < item.index("request(c0, true);")   # of every warp, for any number of slices
    stale = item[item.index("if (pos_now != pos) {"):item.index("angles();\n    }\n  }\n\n  // ---- 1.")]
    wait, poll, again = (stale.index(x) for x in ("tc::mbar_wait(bar_k, phase,", "tc::mbar_drain(bar_k, phase,", "request(c0, true);"))
    assert wait < stale.index("if (!ok) {") < poll < again and stale[:again].rstrip().endswith("if (ok) {")
    gone = item.index("if (!ok) {  // without keys")
    assert item.rindex("env.sync_cta();", 0, gone) < gone < item.index("for (; c0 < t1; c0 += 4 * KT)")
    assert "c0 = t1;" in item[gone:gone + 120]


def test_cleared_rows_of_a_tile_come_before_its_next_load():
    """Ordinary stores to a tile and TMA's next writes to it are different proxies: without a fence the stores may come last."""
    text = open(os.path.join(CSRC, "attn_decode.cuh")).read()
    clear = text.index("*chunk_of(vw, live + i / CH, i % CH) = make_uint4")
    fence = text.index("if (c0 + 4 * KT < t1) asm volatile(\"fence.proxy.async.shared::cta;\"", clear)
    assert clear < fence < text.index("__syncwarp();", fence) < text.index("request(c0 + 4 * KT, false);")


def test_decode_attention_checks_what_it_takes_from_the_device():
    """Slots and positions come from device memory: one out of range raises the error word and appends nothing.  The environment
    holds what it needs by value, not the address of a kernel parameter."""
    text = open(os.path.join(CSRC, "attn_decode.cu")).read()
    env = text[text.index("struct KernelEnv {"):text.index("__global__")]
    assert "AttnDecArgs" not in env and "= &a;" not in kernel("attn_decode.cu", "k_attn_dec")
    item = open(os.path.join(CSRC, "attn_decode.cuh")).read()
    slot, settled = item.index("place = a.rows.slot[b];"), item.index("int64_t pos_now = env.settle(pos);")
    for at, before in ((slot, "kbase ="), (settled, "if (pos_now != pos)")):
        check = item[at:item.index(before, at)]
        assert "*a.err = DEV_INDEX;" in check and "in_range = false;" in check
    assert "(place + 1) * a.nkv * a.Tmax > a.cache_rows" in item and "(uint64_t)pos_now >= (uint64_t)a.Tmax" in item
    assert "if (id >= rep && split == 0 && in_range) put(" in item and item.count("split == 0") == 1
