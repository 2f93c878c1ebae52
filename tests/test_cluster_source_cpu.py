"""Every kernel that touches another CTA's shared memory first waits until all CTAs of its cluster run (CUDA requires
that all thread blocks have started before their distributed shared memory is accessed).  Read from the sources: a
missing wait seldom shows on a device."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcnla_b200", "csrc")
WAIT = re.compile(r"\bcluster_sync\(|\.sync\(\)|barrier_wait\(|barrier\.cluster\.wait")


def _accesses():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = open(path).read()
        for m in re.finditer(r"map_shared_rank\(", src):
            body = src.rfind("\n__global__", 0, m.start())          # the kernel the access is in
            yield os.path.basename(path), src.count("\n", 0, m.start()) + 1, src[body:m.start()]


@pytest.mark.parametrize("name,line,before", [pytest.param(*a, id="%s:%d" % a[:2]) for a in _accesses()])
def test_cluster_has_started_before_remote_shared_memory(name, line, before):
    assert before.lstrip().startswith("__global__"), "no kernel found around %s:%d" % (name, line)
    assert WAIT.search(before), "%s:%d" % (name, line)


def _mma_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for body in re.split(r"\n(?=__global__)", open(path).read())[1:]:
            if "tcgen05.alloc" in body:
                yield os.path.basename(path), body


@pytest.mark.parametrize("name,body", [pytest.param(*k, id=k[0]) for k in _mma_kernels()])
def test_no_mma_or_copy_outlives_its_cta(name, body):
    """Whatever wait ran out: the issuer commits what it issued and waits for it (bounded), and the producer waits for
    its copies, before tensor memory and shared memory go back."""
    issuer = body[body.index("MMA issuer"):body.index("tcgen05.dealloc")]
    last = issuer.rindex("umma_commit(")
    assert issuer[last:].startswith("umma_commit(&mma_done)") and "mbar_wait(&mma_done, 0)" in issuer[last:]
    producer = body[body.index("---- producer"):body.index("MMA issuer")]
    assert "mbar_wait(&full" in producer[producer.index("issued"):]
