"""A grid barrier that gives up ends the refine with a status, and the session, the
other teams and the GPU go on. The kernels of k <= 32 are compiled a second time
with a wait that runs out at the first look; every wait still ends by itself."""
import pytest

from variant import run_with_variant

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import sys
import numpy as np
import lpgpu as lp
from lpgpu import gen

lp.LIB_PATH = sys.argv[1]
cfg, pipeline = lp.default_config(), lp.default_config(flags=lp.FLAG_MULTI_LAUNCH)


def status(call):
    try:
        call()
    except lp.LpgpuError as e:
        return e.status
    return lp.OK


for n, k in ((20000, 6), (131071, 2)):
    inst = gen.random_small(n, n=n, m=n, k=k)
    with lp.Session(0) as s:
        s.upload(inst.hg)
        for _ in range(2):
            s.set_partition(k, inst.part, eps=0.03)
            assert status(lambda: s.refine(cfg)) == lp.ERR_TIMEOUT
            assert status(lambda: s.metrics()) == lp.ERR_STATE  # the partition is half moved
        s.set_partition(k, inst.part, eps=0.03)
        r = s.refine(pipeline)
        assert r.km1_after < r.km1_before and s.metrics()[0] == r.km1_after
        want = s.partition()
    with lp.Session(0) as s:
        s.upload(inst.hg)
        s.set_partition(k, inst.part, eps=0.03)
        s.refine(pipeline)
        assert np.array_equal(s.partition(), want)
# clusters meet in hardware and have no such limit
inst = gen.random_small(5, n=5000, m=5000, k=6)
parts = []
for c in (cfg, pipeline):
    with lp.Session(0) as s:
        s.upload(inst.hg)
        s.set_partition(6, inst.part, eps=0.03)
        s.refine(c)
        parts.append(s.partition())
assert np.array_equal(*parts)
print("ok")
"""


def test_a_grid_barrier_that_gives_up_ends_the_refine(lp, tmp_path):
    run_with_variant(tmp_path, "team_w1.cu", ["-DLPGPU_TEAM_WAIT_CLOCKS=0ll", "-DLPGPU_TEAM_WAIT_POLLS=1u"], PROGRAM)
