"""The failure path of the emulated-FP64 update without a GPU: which copies and MMA batches are
still in flight when it gives up (cuda/oz_pipeline.hpp, run by a C++ program against a model of
the barriers), and that the kernel waits for them."""
import json
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "soverign-gpu-accelerator-_gb300", "csrc")


def test_phases(tmp_path):
    exe = os.path.join(str(tmp_path), "oz_pipeline")
    p = subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CSRC,
                        os.path.join(HERE, "cpp", "oz_pipeline.cpp"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.stdout, p.stderr)
    res = json.loads(p.stdout)
    assert res["failed"] == 0 and res["checks"] > 100000
    assert res["fixed_parity_leaves"] > 1000            # a wait with a fixed parity ends too early


def _kernel(name):
    src = open(os.path.join(CSRC, "cuda", "kkt_engine.cu")).read()
    body = src[src.index(name + "(StepArgs"):]
    return re.sub(r"//.*", "", body[:body.index("\n}\n")])


def test_the_kernel_waits_for_what_it_issued():
    body = _kernel("k_update_oz")
    # every copy and every batch of MMAs is logged where it is issued, and waited for at the end
    assert body.count("oz_copy_rows(") == body.count("copies.start(") == 2
    assert body.count("oz_commit(") == body.count("batches.start(") == 2
    assert "copies.last_parity(b)" in body and "batches.last_parity(b)" in body
