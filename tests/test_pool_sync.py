"""The warps' cone pools (march_kernel.cuh): a count in shared memory that one lane writes and others append behind
needs a warp barrier between the two, since votes and shuffles order no memory."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "project-marshmallow_gb300", "csrc")


def test_plain_writes_of_the_count_are_behind_a_barrier():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "march_kernel.cuh")).read())
    writes = [m.end() for m in re.finditer(r"\bwaiting\s*\[[^\n]*\]\s*[-+]?=[^=][^;]*;", src)]
    assert len(writes) == 2  # the reset and a round's take
    for at in writes:
        assert re.match(r"\s*__syncwarp\(\);", src[at:]), src[at - 80:at + 80]


def test_every_march_with_a_pool_resets_it():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "march_kernel.cuh")).read())
    appends = [m.start() for m in re.finditer(r"atomicAdd\(&q\.waiting", src)]
    resets = [m.start() for m in re.finditer(r"\bpool_reset\(q\);", src)]
    assert len(appends) == len(resets) == 2
    assert resets[0] < appends[0] < resets[1] < appends[1]
