"""The blocks of a BFS cluster end together when the wait of one of them runs
out: nobody uses the shared memory of a block that is gone, and every block
(the one that reports among them) knows.  The kernel's end protocol is compiled
for the host and run with a thread per block."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cluster") / "model")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread",
                    "-I" + os.path.join(ROOT, "graph_analytics_applesilicon_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "cluster_leave_model.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("notices", [0, 1])
@pytest.mark.parametrize("blocks,quitter,at", [(2, 0, 0), (2, 1, 2), (4, 3, 1), (8, 0, 3), (16, 15, 0), (16, 7, 2), (8, -1, 0)])
def test_nobody_uses_a_block_that_is_gone(model, blocks, quitter, at, notices):
    if quitter <= 0 and notices:
        pytest.skip("block 0 is the one that does not wait")
    r = subprocess.run([model, str(blocks), "5", str(quitter), str(at), str(notices)], check=True, timeout=60,
                       capture_output=True, text=True)
    assert r.stdout.split() == ["0", "0", "0"]  # strayed uses, blocks that did not report, blocks left behind
