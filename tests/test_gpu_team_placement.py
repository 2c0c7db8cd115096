"""Where a team cannot be placed (a partition of the GPU too small for a cluster or
a cooperative grid) the refine takes the pipeline, or one CTA when its form is
settled. The library is linked a second time with a limit on the team in place of
such a partition, and runs in a process of its own."""
import pytest

from variant import run_with_variant

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import sys
import numpy as np
import lpgpu as lp
from lpgpu import gen

lp.LIB_PATH = sys.argv[1]
most = int(sys.argv[2])
assert lp.lib()._name == sys.argv[1]


def refine(insts, k, flags):
    with lp.Session(0) as s:
        if len(insts) == 1:
            s.upload(insts[0].hg)
            s.set_partition(k, insts[0].part, eps=0.03)
        else:
            s.upload_batch([x.hg for x in insts])
            s.set_partition_batch([k] * len(insts), [x.part for x in insts], eps=0.03)
        before = lp.kernel_launches()
        r = s.refine(lp.default_config(flags=flags))
        launches = lp.kernel_launches() - before
        part = s.partition()
        return launches, part if isinstance(part, np.ndarray) else np.concatenate(part), r.km1_after, r.moves


# vertices, instances, CTAs of the default team
for n, count, team in ((1500, 1, 1), (5000, 1, 16), (20000, 1, 152), (5000, 2, 8)):
    insts = [gen.random_small(n + i, n=n, m=n, k=6) for i in range(count)]
    want = refine(insts, 6, lp.FLAG_MULTI_LAUNCH)
    for flags in (0, lp.FLAG_PERSISTENT):
        got = refine(insts, 6, flags)
        assert np.array_equal(got[1], want[1]) and got[2:] == want[2:], (n, count, flags)
        one_launch = flags or team <= most
        assert (got[0] < 10) == bool(one_launch), (n, count, flags, got[0], want[0])

# stepped rounds shrink their teams
insts = [gen.random_small(50 + i, n=5000, m=6000, k=5) for i in range(2)]
alone = [refine([x], 5, lp.FLAG_MULTI_LAUNCH) for x in insts]
sessions = [lp.Session(0).upload(x.hg) for x in insts]
for s, x in zip(sessions, insts):
    s.set_partition(5, x.part, eps=0.03)
    s.begin_rounds(lp.default_config())
stepper, running = lp.Stepper(), list(sessions)
while running:
    done = stepper.round(running)
    running = [s for s, d in zip(running, done) if not d]
for s, a in zip(sessions, alone):
    assert s.end_rounds().km1_after == a[2]
    assert np.array_equal(s.partition(), a[1])
print("ok")
"""


@pytest.mark.parametrize("most", [1, 4, 16])
def test_refines_without_room_for_their_team(lp, tmp_path, most):
    run_with_variant(tmp_path, "team.cu", ["-DLPGPU_TEAM_MOST=%d" % most], PROGRAM, str(most))
