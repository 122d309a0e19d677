"""CPU: a kernel may touch another CTA's shared memory only once that CTA is known
to run, that is after a cluster barrier.  Read from the sources."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "lineax_gb300" / "csrc"
# a value loaded or stored through a mapped address; taking the address alone is no access
ACCESS = re.compile(r"\*\s*(?:cluster\.map_shared_rank|remote)\s*\("
                    r"|(?:cluster\.map_shared_rank|remote)\([^;]*?\)\s*\[")
BARRIER = re.compile(r"cluster\.(?:sync|barrier_wait)\(\)")


def inline_lambdas(text):
    """Each local lambda's body at the place of its first call."""
    for m in reversed(list(re.finditer(r"auto (\w+) = \[&\]\([^)]*\)[^{;]*\{", text))):
        end, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        body, text = text[m.end():end - 1], text[:m.start()] + text[end:]
        call = re.compile(r"\b%s\(" % m.group(1)).search(text, m.start())
        if call:
            text = text[:call.start()] + body + text[call.start():]
    return text


def kernels():
    found = []
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for part in re.split(r"__global__", text)[1:]:
            part = part.split("\nstatic ")[0]
            if "map_shared_rank" in part:
                name = re.search(r"(\w+_kernel)\(", part).group(1)
                found.append(pytest.param(inline_lambdas(part), id=name))
    return found


@pytest.mark.parametrize("body", kernels())
def test_remote_access_after_a_cluster_barrier(body):
    access, barrier = ACCESS.search(body), BARRIER.search(body)
    assert barrier is not None
    assert access is None or barrier.start() < access.start(), body[access.start():][:80]
