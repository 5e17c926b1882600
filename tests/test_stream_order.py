"""Kernels launched as programmatic dependents start while the kernel ahead of them still
runs.  Whatever follows one in the stream waits for it alone, so it has to wait itself, and
it may let its successor in only after that."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "winnow_b200" / "csrc"
WAIT = re.compile(r"griddepcontrol\.wait|\bgriddep_wait\(\)|\bbegin_rotation\(\)")
TRIGGER = re.compile(r"griddepcontrol\.launch_dependents|\bgriddep_launch\(\)")


def kernels(text):
    """name -> body of every __global__ function."""
    found = {}
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
        at = text.index("{", m.end())
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        found[m.group(1)] = text[at:end]
    return found


def dependents(text):
    """Names of the kernels a file launches with the programmatic attribute."""
    if "cudaLaunchAttributeProgrammaticStreamSerialization" not in text:
        return set()
    names = set(re.findall(r"cudaLaunchKernelEx\(&cfg, (?:\w+::)?(\w+)", text))
    if "kernel" in names:
        names.discard("kernel")
        names |= set(re.findall(r"auto kernel = (?:\w+::)?(\w+)", text))
        names |= set(re.findall(r"\b(?:fixed|general)\((\w+)<", text))
    return names


def test_programmatic_dependents_wait_before_they_let_others_in():
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        bodies = kernels(text)
        for name in dependents(text):
            waits = [m.start() for m in WAIT.finditer(bodies[name])]
            triggers = [m.start() for m in TRIGGER.finditer(bodies[name])]
            assert waits, f"{path.name}: {name} never waits for the kernel ahead of it"
            assert all(t > waits[-1] for t in triggers), f"{path.name}: {name} lets its successor in before it has waited"
            seen += 1
    assert seen >= 12
