"""Rules of the CUDA sources that only a failure on the device would show, checked in the text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pretrained_rstr_b200", "csrc")


def _code(name):
    """A source without its comments."""
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)


def test_warps_meet_before_the_aligned_cluster_barrier_of_the_split_product():
    """barrier.cluster.*.aligned wants whole warps: in the cluster split-K product a bounded wait may
    end differently for a warp's lanes, so the answer is the warp's and the warp meets again."""
    kernel = _code("gemm_bf16_midm.cu").split("gemm_midm_kernel(Args", 1)[1].split("midm_smem()", 1)[0]
    assert re.search(r"alive = __all_sync\(0xffffffffu, mbar_wait\(", kernel)
    for barrier in ("cluster_wait();", "cluster_arrive();"):
        for before in kernel.split(barrier)[:-1]:
            last = [line.strip() for line in before.strip().split("\n") if not line.strip().startswith("MT_TRACE")][-1]
            assert last in ("__syncwarp();", "cluster_arrive();", "prb_grid_launch_dependents();"), last


def test_a_warp_of_the_ring_attention_has_one_answer_to_a_wait():
    """Its loop goes on with shuffles and matrix instructions of whole warps: a lane may not leave alone."""
    waits = re.findall(r"if \(!(.*)mbar_wait_bounded", _code("attention_decode_ring.cuh"))
    assert waits and all(w == "__all_sync(0xffffffffu, " for w in waits)


def test_a_wait_that_gave_up_in_a_32_bit_tile_stops_its_whole_cluster():
    """A bounded wait may end differently for a CTA's threads: who requests copies has waited for the stage's last
    one, whoever gave up the status is recorded, and no CTA of the cluster stores sums that hold the broken part."""
    kernel = _code("gemm_f32.cu").split("gemm_f32_tile_kernel(Args", 1)[1].split("int launch_tile_by", 1)[0]
    requests, rest = kernel.split("prb_grid_wait();", 1)
    assert re.search(r"if \(tid == 0 && alive\) \{[^}]*mbar_expect_tx", requests)
    chunk = rest.split("mbar_wait(", 1)[1].split("load_rows(c + TILE_STAGES", 1)[0]
    assert re.search(r"alive = false;\s*for \(int i = c; tid == 0 && i < min\(c1, c \+ TILE_STAGES\); \+\+i\)\s*"
                     r"for \(uint32_t w = 0; w < tc5::WAIT_LIMIT", chunk)
    assert re.search(r"__syncthreads\(\);\s*$", chunk)             # every thread's reads are behind the next request
    assert re.search(r"tid == 0 && \*failed\) \{\s*prb_set_status\(p.status, PRB_S_WAIT_TIMEOUT", rest)
    before, store = rest.split("cluster_sync_all();", 1)
    assert "PRB_S_WAIT_TIMEOUT" in before and "finish(p" not in before
    assert re.search(r"any \|= ld_cluster1\(smem_u32\(&failed_word\), q\);\s*alive = any == 0;", store.split("finish(p", 1)[0])
    assert "if (row >= p.m || !alive) continue;" in store


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_a_wait_names_the_phase_it_waits_for(name):
    """A barrier answers at once for one of the two parities: a loop that takes either waits for nothing,
    and a kernel that gave up would leave with copies on their way into its shared memory."""
    assert not re.search(r"try_wait\([^;]*,\s*0\)\s*\|\|[^;]*try_wait\([^;]*,\s*1\)", _code(name))


@pytest.mark.parametrize("name", ["gemm_f32.cu", "attention_f32.cu"])
def test_no_launch_sets_a_kernel_attribute(name):
    """cudaFuncSetAttribute costs the host as much as a launch of the small kernels of a decode step."""
    code = _code(name)
    assert "cudaFuncSetAttribute" not in code and "prb_allow_shared<" in code


def test_float32_products_share_no_switch_between_threads():
    """Which kernel a product takes is its call's own argument: no variable of the file that other threads' launches
    read as well."""
    assert not re.search(r"^(static\s+)?(int|bool|long)\s+g_\w+\s*(=|;)", _code("gemm_f32.cu"), flags=re.M)


def test_the_first_kernel_behind_the_page_copies_is_launched_the_plain_way():
    """The decode attention asks for cached pages before the kernel ahead of it has ended: all that follows the page
    copies of a step may start early only because the embedding, and the copies themselves, do not."""
    code = _code("elementwise.cu")
    for entry in ("prb_embed(", "prb_copy_pages("):
        body = code.split("PRB_API int " + entry, 1)[1].split("PRB_API", 1)[0]
        assert "<<<" in body and "prb_launch" not in body
