"""Distributed shared memory in the kernels' sources: CUDA lets a CTA touch
another CTA's shared memory only once every CTA of the cluster is known to run,
so a kernel waits at a cluster barrier before its first remote access (its own,
or one in a function that it calls), and no CTA may leave while another can
still reach it, so a cluster barrier also follows the last one.  Read from the
source: an access that breaks this is never run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "argus-sdr_b200", "csrc")
WAIT = re.compile(r"\.sync\s*\(\s*\)|barrier_wait\s*\(|barrier\.cluster\.wait")
REMOTE = re.compile(r"map_shared_rank\s*\(|\bmapa\.")


def _code(path):
    """The source without comments."""
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", " ", text, flags=re.S)


def _functions(text):
    """(name, body, is a kernel) of every function definition."""
    for m in re.finditer(r"(__global__|__device__)[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*\{", text):
        name = next((w for w in re.findall(r"\b(\w+)\s*\(", m.group(0)) if not w.startswith("__")), m.group(2))
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield name, text[m.end():at - 1], m.group(1) == "__global__"


def _kernels():
    """(file, kernel, body, pattern of its remote accesses) of the kernels with any."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        funcs = list(_functions(_code(os.path.join(CSRC, f))))
        remote = {n for n, body, kernel in funcs if not kernel and REMOTE.search(body)}
        call = "|".join([REMOTE.pattern] + [rf"\b{n}\s*\(" for n in sorted(remote)])
        for name, body, kernel in funcs:
            if kernel and re.search(call, body):
                yield pytest.param(body, call, id=f"{f}:{name}")


def test_the_solver_is_among_them():
    assert any("k_pll_newton" in p.id for p in _kernels())


@pytest.mark.parametrize("body,remote", list(_kernels()))
def test_cluster_wait_before_the_first_and_after_the_last_remote_access(body, remote):
    at = [m.start() for m in re.finditer(remote, body)]
    waits = [m.start() for m in re.finditer(WAIT, body)]
    assert waits and min(waits) < at[0], "remote shared memory before the cluster is known to run"
    assert max(waits) > at[-1], "a CTA may leave while its shared memory is still in use"
