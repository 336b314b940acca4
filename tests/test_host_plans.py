"""The FP32 launch plan on the host (tests/host_cuda/plans.cpp): a front is updated
two-level by its own size, whatever it is batched with, and only fronts and K
blocks with columns to update get scaled rows."""
from test_host_lifetimes import build, run


def test_two_level_fronts(tmp_path):
    p = run(build(tmp_path, "plans"))
    assert p.returncode == 0 and p.stdout == "0\n", p.stdout + p.stderr[-3000:]
