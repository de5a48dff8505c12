"""dpb_sumcheck_begin_partial: the ranks' parts of a term list may be of different forms, and each rank's part takes the
kernels of its own form.  The ranks' messages and final evaluations equal the oracle's over the union of the lists."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def comm_dir(tmp_path_factory):
    out = tmp_path_factory.mktemp("comm")
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-Wall", "-shared", "-fPIC", os.path.join(ROOT, "tests", "one_gpu_comm.c"), "-I",
                    os.path.join(CUDA, "include"), "-L", os.path.join(CUDA, "lib64"), "-lcudart", "-Wl,-soname,libnccl.so.2",
                    "-o", str(out / "libnccl.so.2")], check=True)
    return str(out)


@pytest.mark.gpu
@pytest.mark.parametrize("field", ["gl", "fr"])
@pytest.mark.parametrize("case", ["padded", "product", "eq"])
@pytest.mark.parametrize("n,exchange", [(4, "shared"), (13, "shared"), (13, "nccl"), (16, "shared")])
def test_parts_of_different_forms(comm_dir, field, case, n, exchange):
    env = dict(os.environ, LD_LIBRARY_PATH=comm_dir + ":" + os.environ.get("LD_LIBRARY_PATH", ""))
    if exchange == "nccl":
        env["DPB_NO_SHARED_EXCHANGE"] = "1"
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "partial_ranks.py"), field, str(n), case, exchange], cwd=ROOT,
                       env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("equal"), r.stdout[-2000:] + r.stderr[-3000:]
