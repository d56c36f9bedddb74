"""Index arithmetic of the layout header at the ends of its range, compiled for
the host: states of that size do not fit a test."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nexus_b200", "csrc")


def _run(tmp_path, body):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include "nxm_layout.h"\n#include <cstdio>\nusing namespace nxm;\nint main() {\n' + body + "\n}\n")
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


def test_node_words_of_the_last_blocks(tmp_path):
    """The gather P2G stores single words; a block's words follow the block before's up to kMaxBlocks."""
    blocks = [0, 1, (1 << 24) - 1, 1 << 24, (1 << 24) + 5, int(_run(tmp_path, 'printf("%u", kMaxBlocks);')[0]) - 1]
    got = _run(tmp_path, "".join(f'printf("%zu %zu ", node_word({b}u, 0u), node_word({b}u, 255u));' for b in blocks))
    assert [int(x) for x in got] == [v for b in blocks for v in (b * 256, b * 256 + 255)]
    det = open(os.path.join(CSRC, "nxm_transfer_det.cu")).read()
    assert "* 256u" not in det  # no word index formed in 32 bits beside it


def test_node_loops_end_at_the_last_block(tmp_path):
    """`for (t = thread; t < blocks * 64; t += stride)` in 32 bits: the first t past the end must not wrap
    to a small one, or the loop starts again and never ends."""
    blocks = int(_run(tmp_path, 'printf("%u", kMaxBlocks);')[0])
    stride = 148 * 16 * 256  # the largest launch over nodes
    assert blocks * 64 + stride <= 1 << 32
    assert blocks * 64 + 63 < (1 << 32) - 1  # the last cell's key is not NONE


def test_records_of_in_place_kernels_are_not_read_as_read_only():
    """Deterministic and CPIC steps write the records they read: the read-only path
    (ld.global.nc, __ldg) is only for arrays that a kernel does not write."""
    for name in ("nxm_device.cuh", "nxm_transfer.inc.cuh", "nxm_transfer_det.cu"):
        text = open(os.path.join(CSRC, name)).read()
        assert "ld.global.nc" not in text, name
        for record in ("in.kin", "in.aff", "in.tail", "in.def", "in.mat", "in.pstate", "out."):
            assert f"__ldg(&P.{record}" not in text, (name, record)
