"""bench.py takes ncu figures only from summaries of the present kernels."""

import os
import shutil

import bench

SUMMARY = "# A summary\n\nl2_bytes_per_ray: 696.1\nlanes_per_instruction: 17\n"


def test_figures_of_another_kernel_are_left_out(tmp_path):
    def read(text, code="abc123"):
        (tmp_path / "s.md").write_text(text)
        return bench.profile_figures("s.md", folder=str(tmp_path), code=code)
    want = {"l2_bytes_per_ray": 696.1, "lanes_per_instruction": 17.0}
    assert read(SUMMARY + "code: abc123\n") == want
    assert read(SUMMARY + "code: 000000\n") == {}
    assert read(SUMMARY) == {}  # captured before summaries named their code
    assert bench.profile_figures("none.md", folder=str(tmp_path), code="abc123") == {}


def test_digest_follows_code_not_comments(tmp_path):
    csrc = os.path.join(bench.ROOT, "sundog_b200", "csrc")
    shutil.copytree(csrc, tmp_path / "csrc")
    was = bench.code_digest(csrc)
    f = tmp_path / "csrc" / "wavefront.cu"
    text = f.read_text()
    f.write_text("// a comment\n" + text + "\n/* and\n another */\n")
    assert bench.code_digest(str(tmp_path / "csrc")) == was
    f.write_text(text.replace("#define SDB_WF_FETCH_IDLE 20", "#define SDB_WF_FETCH_IDLE 24"))
    assert bench.code_digest(str(tmp_path / "csrc")) != was
