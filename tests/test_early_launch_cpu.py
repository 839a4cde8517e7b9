"""Rules of the kernels that start under the launch in front of them, read off their source:

- one that claims tensor memory lets the next launch start only when it has its own.  That launch may claim tensor memory as well and
  keeps it until this one has ended, and an allocation waits without a limit;
- what an earlier launch writes does not come through ``const ... __restrict__`` pointers: the compiler may move such loads in
  front of the wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hf2q_b200" / "csrc"
CODE = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}
TRIGGER = re.compile(r"pdl_trigger\(\)|griddepcontrol\.launch_dependents")
WAIT = re.compile(r"pdl_wait\(\)|griddepcontrol\.wait")


def closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def functions(text):
    """(is a kernel, name, parameters, body) of the device functions of a file"""
    for head in re.finditer(r"__(global|device)__", text):
        rest = re.compile(r"(?:__launch_bounds__\s*(\())|([A-Za-z_]\w*)\s*\(|[;{=]").match
        at = head.end()
        while at < len(text):
            m = rest(text, at)
            if m is None:
                at += 1
            elif m.group(1):
                at = closing(text, m.start(1), "()") + 1
            elif m.group(2):
                end = closing(text, m.end() - 1, "()")
                brace = re.compile(r"\s*(?:const)?\s*\{").match(text, end + 1)
                if brace:
                    yield head.group(1) == "global", m.group(2), text[m.end():end], text[brace.end() - 1:closing(text, brace.end() - 1, "{}") + 1]
                break
            else:
                break


ALL = [(file, *f) for file, text in CODE.items() for f in functions(text)]
EARLY = [(file, name) for file, kernel, name, _, body in ALL if kernel and WAIT.search(body)]


def test_the_source_is_read():
    names = {name for _, name in EARLY}
    assert {"gemm_tc_kernel", "dense_gemm_tc_kernel", "window_prefill_tc_kernel", "window_prefill_f32_kernel", "dense_matvec_kernel", "gemv_mma_kernel"} <= names
    assert sum(kernel and "tmem_alloc(" in body for _, kernel, _, _, body in ALL) == 4


@pytest.mark.parametrize("file,name", [(file, name) for file, kernel, name, _, body in ALL if kernel and "tmem_alloc(" in body])
def test_tensor_memory_is_claimed_before_the_next_launch_may_start(file, name):
    body = next(b for f, _, n, _, b in ALL if (f, n) == (file, name))
    owned = body.index("__syncthreads()", body.index("tmem_alloc("))
    assert all(m.start() > owned for m in TRIGGER.finditer(body))


@pytest.mark.parametrize("file,name", EARLY)
def test_what_earlier_launches_write_is_not_taken_for_read_only(file, name):
    todo, seen = [name], set()
    while todo:
        n = todo.pop()
        for f, _, fn, params, body in ALL:
            if fn != n or (f, fn, params) in seen or not (f == file or f.endswith(".cuh")):
                continue
            seen.add((f, fn, params))
            for p in re.findall(r"const[^,*]*\*\s*__restrict__\s*(\w+)", params):
                assert p in ("w", "b"), f"{fn}: {p}"                        # weights, blocks of them
            todo += set(re.findall(r"\b([a-z_]\w*)\s*(?:<[^;{}()]*>)?\s*\(", body))
