"""Blocks of a cluster may touch each other's shared memory only once all of
them are known to run, and a block may leave only when nobody will touch its
memory any more: every kernel body that maps another block's shared memory
arrives at and waits on the cluster barrier on every thread's path before its
first access, and waits again after its last (read from the source: a missing
wait is a race, which no run can be relied on to show)."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lammps-lbm-psm_gb300", "csrc")
WAIT = re.compile(r"barrier_wait\(|this_cluster\(\)\.sync\(|cluster\.sync\(")


def bodies():
    """(file, body) of every function that maps another block's shared memory."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"^(?:template|static|__global__|inline)[^;{}]*\{", src, re.M):
            depth, k = 1, m.end()
            while depth and k < len(src):
                depth += {"{": 1, "}": -1}.get(src[k], 0)
                k += 1
            if "map_shared_rank" in src[m.end():k]:
                yield os.path.basename(path), src[m.end():k]


def depth_at(body, pos):
    """Loops and branches around a position (braces opened and not closed)."""
    return body[:pos].count("{") - body[:pos].count("}")


CASES = list(bodies())
EACH = pytest.mark.parametrize("name,body", CASES, ids=[f for f, _ in CASES])


def test_there_is_such_a_kernel():
    assert [f for f, _ in CASES] == ["particles.cu"]


@EACH
def test_wait_before_the_first_remote_access(name, body):
    first = body.index("map_shared_rank")
    waits = [m.start() for m in WAIT.finditer(body) if m.start() < first]
    # outside every loop and branch in braces, so that all threads take part
    assert [w for w in waits if depth_at(body, w) == 0], name


@EACH
def test_wait_after_the_last_remote_access(name, body):
    assert WAIT.search(body, body.rindex("map_shared_rank")), name


@EACH
def test_every_split_wait_has_its_arrival(name, body):
    arrive = [m.start() for m in re.finditer(r"barrier_arrive\(", body)]
    wait = [m.start() for m in re.finditer(r"barrier_wait\(", body)]
    assert len(arrive) == len(wait) and all(a < w for a, w in zip(arrive, wait)), name
    assert all(depth_at(body, p) == 0 for p in arrive + wait), name
