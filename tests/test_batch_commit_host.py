"""Memory of a batch's commit, on the CPU: the C host layer linked against a
fake CUDA layer (tests/c/test_batch_commit.c), where allocations and captures
fail on request and a launched job that points into freed memory is seen."""
import os
import subprocess

import pytest

from conftest import ROOT
from vkhel_gb300 import workloads

CSRC = os.path.join(ROOT, "vkhel_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("batch_commit") / "test_batch_commit")
    host = [os.path.join(CSRC, f + ".c") for f in ("api", "batch", "tables", "numbers", "tuning")]
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-g", "-Wall", "-Wextra", "-Wno-unused-parameter", "-pthread",
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "c", "test_batch_commit.c"),
                    *host, "-o", exe, "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["composed_where_there_is_room", "retry_without_scratch",
                                      "retry_with_other_tuning",
                                      "no_room_beside_the_table", "budget_for_a_later_vector"])
def test_batch_commit(program, scenario):
    n = 1 << 17
    q = workloads.ntt_primes(n, 1)[0]
    r = subprocess.run([program, scenario, str(q), str(workloads.root_for(n, q))], capture_output=True, text=True,
                       env=dict(os.environ, VKHEL_TUNE_TABLE=""))
    assert r.returncode == 0, r.stderr
