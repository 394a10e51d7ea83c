"""Linked launches (csrc/pic_device.cuh, launch_linked): a linked kernel's blocks
are resident while the launch before still writes what they will read, so the
kernel waits for that launch before it touches memory, and reads it by loads
that the wait orders: never through the read-only path, whose data must not
change during the kernel's life, and never by an asm the compiler may move."""

import re
from pathlib import Path

import pytest

from goldens import pkg

CSRC = Path(pkg().__file__).parent / "csrc"


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _body(code, name):
    """The body of kernel `name`."""
    at = re.search(r"__global__[^;{]*\b" + name + r"\s*\([^{;]*\)\s*\{", code)
    assert at, name
    depth, end = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        end += 1
    return code[at.end() : end]


def _linked():
    found = set()
    for path in CSRC.glob("*.cu"):
        for name in re.findall(r"\blaunch_linked\(\s*(\w+)", _code(path)):
            found.add((path.name, name))
    return sorted(found)


def test_there_are_linked_kernels():
    assert {"step_kernel", "wide_step_kernel", "batched_step_kernel", "wide_adjoint_kernel",
            "adjoint_fold_kernel"} == {name for _, name in _linked()}


@pytest.mark.parametrize("file,name", _linked())
def test_a_linked_kernel_waits_before_it_touches_memory(file, name):
    body = _body(_code(CSRC / file), name)
    before = body[: body.index("wait_for_prev();")]
    # declarations of shared memory and locals only
    assert not re.search(r"\b(for|while|if)\b|load|->|\*\s*\w+\s*[;=)]|=[^;]*\[", before), before


@pytest.mark.parametrize("path", sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh")), ids=lambda p: p.name)
def test_no_load_takes_the_read_only_path(path):
    code = _code(path)
    assert not re.search(r"\b__ldg\s*\(|ld\.global\.nc", code)
    for asm in re.findall(r"\basm\s*(volatile)?\s*\(\s*\"([^\"]*)", code):
        if re.match(r"\s*ld\.", asm[1]):
            assert asm[0] == "volatile", asm[1]
