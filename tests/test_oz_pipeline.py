"""The failure path of the emulated-FP64 update without a GPU: which copies and MMA batches are
still in flight when it gives up, and that its warps enter the diagonal tile together or not at
all (cuda/oz_pipeline.hpp, run by a C++ program against a model of the barriers); and that the
kernel keeps to both."""
import json
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "soverign-gpu-accelerator-_gb300", "csrc")


def test_phases_and_joins(tmp_path):
    exe = os.path.join(str(tmp_path), "oz_pipeline")
    p = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + CSRC,
                        os.path.join(HERE, "cpp", "oz_pipeline.cpp"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.stdout, p.stderr)
    res = json.loads(p.stdout)
    assert res["failed"] == 0 and res["checks"] > 100000
    assert res["fixed_parity_leaves"] > 1000            # a wait with a fixed parity ends too early
    assert res["together"] > 1000 and res["apart"] > 100


def _kernel(name):
    src = open(os.path.join(CSRC, "cuda", "kkt_engine.cu")).read()
    body = src[src.index(name + "(StepArgs"):]
    return re.sub(r"//.*", "", body[:body.index("\n}\n")])


def test_the_kernel_waits_for_what_it_issued():
    body = _kernel("k_update_oz")
    # every copy and every batch of MMAs is logged where it is issued, and waited for once every
    # warp is through, if any of them gave up
    assert body.count("oz_copy_rows(") + body.count("oz_commit(") == body.count("issued.start(") == 4
    end = body[body.rindex("__syncthreads();"):]
    assert re.search(r"if \(\*fail != 0 && wid >= 8\)", end) and "issued.last_parity(b)" in end
    assert end.index("issued.last_parity(b)") < end.index("tcgen05.dealloc")
    # the barriers without a limit are reached by all of the eight warps that joined, or by none
    assert "bar.sync" not in body and body.count("tile_sync()") == body.count("potrf_tile(") == 1
    assert re.search(r"in = join\(tri,.*?if \(__shfl_sync\(0xffffffffu, in, 0\)\) \{\s*tile_sync\(\);\s*potrf_tile\(",
                     body, re.S)
    assert "left = leave(tri, swap_joined)" in body
