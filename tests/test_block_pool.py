"""Page-locked host memory comes from a bounded pool (cuda/block_pool.hpp): its rules, on a counting
backend without a GPU; and that the handles take it from there, since locking and unlocking
pages costs a short-lived one more than its work."""
import json
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "soverign-gpu-accelerator-_gb300", "csrc")


def test_pool(tmp_path):
    exe = os.path.join(str(tmp_path), "block_pool")
    p = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + CSRC,
                        os.path.join(HERE, "cpp", "block_pool.cpp"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, (p.stdout, p.stderr)
    assert json.loads(p.stdout)["checks"] > 1000


def test_no_page_locking_per_handle():
    calls = {}
    for f in ("cuda/dev_common.cuh", "cuda/kkt_engine.cu", "cuda/kkt_engine.hpp", "cuda/gnn.cu", "cuda/gnn.hpp",
              "cuda/device_ipm.cu", "cuda/device_qp.cu", "api/sk_dev_api.cpp"):
        src = open(os.path.join(CSRC, f)).read()
        n = sum(src.count(c) for c in ("cudaMallocHost(", "cudaHostAlloc(", "cudaFreeHost(", "cudaHostRegister("))
        if n:
            calls[f] = n
    assert calls == {"cuda/dev_common.cuh": 2}        # the pool's one place to get and to put
