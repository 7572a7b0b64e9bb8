"""What the kernels' sources promise and no run on a healthy GPU would show (CPU)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "htr_b200", "csrc")


def source(path):
    return re.sub(r"//[^\n]*", "", open(path).read()).replace("\\n\\t", " ")


def test_whole_warps_at_aligned_barriers():
    """bar.* and barrier.cluster.*.aligned are undefined where a warp's threads come one by one: each such instruction stands directly behind a
    __syncwarp or another barrier."""
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = source(path)
        for at in re.finditer(r"(?<![\w.])(bar\.(sync|arrive|red)|barrier\.cluster)", text):
            before = text[:text.rindex("asm", 0, at.start())].rstrip()
            assert re.search(r'(__syncwarp\(\);|"barrier\.cluster\.\w+\.\w+\.aligned;" ::: "memory"\);)$', before), (os.path.basename(path), before[-160:])
            found += 1
    assert found >= 10, found


def test_partials_of_the_cluster_are_acquired_from_the_cluster():
    """The inbox of the tensor-core GEMM is filled by other thread blocks: a wait that acquires from its own alone would not order their stores."""
    text = source(os.path.join(CSRC, "packed_gemm_tc.cuh"))
    waits = re.findall(r"mbar_wait(?:_slow)?(<\w+>)?\(smem_u32\(&s_inbox\)", text)
    assert waits and all(w == "<true>" for w in waits)
    assert "mbarrier.try_wait.parity.acquire.cluster.shared::cta" in text


def test_no_thread_block_of_the_gemm_leaves_before_its_transform():
    """A grid whose thread blocks all return without a wait is complete while the launch before it may still run, and later launches wait for
    this grid alone.  The returns of the kernel before its roles begin stand behind a wait."""
    text = source(os.path.join(CSRC, "packed_gemm_tc.cuh"))
    start = text[text.index("packed_gemm_tc_kernel(const GemmParams p)"):]
    start = start[:start.index("tcgen05.alloc")]
    for at in re.finditer(r"\breturn\b", start):
        assert re.search(r'"griddepcontrol\.wait;" ::: "memory"\);\s*$', start[:at.start()]), start[at.start() - 120:at.start()]


def test_pairs_without_an_expert_are_left_before_their_row_is_read():
    """The row of such a pair may never have been written (a gate_up launch skips it too), and reading it costs as much as a pair with work."""
    text = source(os.path.join(CSRC, "gemm_api.cu"))
    kernel = text[text.index("rht_group_kernel(const void*"):]
    assert 0 < kernel.index("if (slot < 0) return;") < kernel.index("load_quad(x")
