"""The order in which kernels take tensor memory and let their successor's blocks come, read from the sources (no GPU).

A successor's block takes its columns before it waits for its predecessor, and ``tcgen05.alloc`` waits without a bound: a kernel that
releases its successor before all of its own blocks hold theirs can wait for columns that come back only when it has ended."""

import re

import pytest

from clockwork_b200.csrc.build import CSRC

RELEASE = re.compile(r"pdl_release\(\)|pdl_enter\(\)|pdl_launch_dependents\(\)|griddepcontrol\.launch_dependents")
BARRIER = re.compile(r"__syncthreads\(\)|cluster_sync\(\)")


def kernels():
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for at in (m.start() for m in re.finditer(r"__global__", text)):
            open_, depth = text.index("{", at), 0
            for end in range(open_, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            body = text[open_:end]
            if "tmem_alloc" in body:
                yield f"{path.name}:{re.search(r'(\w+)\s*\(', text[at + 10 :].split('__launch_bounds__', 1)[-1].split(')', 1)[1]).group(1)}", body


KERNELS = dict(kernels())


@pytest.mark.parametrize("name", KERNELS)
def test_a_kernel_releases_its_successor_only_when_it_holds_its_tensor_memory(name):
    body = KERNELS[name]
    alloc = body.index("tmem_alloc")
    assert body.count("tmem_alloc") == 1
    releases = [m.start() for m in RELEASE.finditer(body)]
    barrier = BARRIER.search(body, alloc)
    assert barrier is not None
    assert all(at > barrier.start() for at in releases), f"{name} releases its successor before every block holds its columns"


def test_all_kernels_that_take_tensor_memory_are_looked_at():
    names = [name.split(":")[0] for name in KERNELS]
    assert sorted(set(names)) == sorted(p.name for p in list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))
                                        if re.search(r"tmem_alloc(_pair)?\(smem", p.read_text()))
