"""Rules of the CUDA sources that no run can show to be kept."""
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paged_batch_engine_b200", "csrc", "kernels")
# what no kernel of a step writes
WEIGHTS = {"table", "pos_table", "gain", "gain1", "gain2", "bias"}


def _closing(text, at, pair="()"):
    depth = 0
    for i in range(at, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def _kernels(text):
    """(name, parameters, body) of every __global__ function that has a body here."""
    for found in re.finditer(r"__global__", text):
        at = found.end()
        while True:
            opened = text.index("(", at)
            name = re.search(r"(\w+)\s*$", text[at:opened]).group(1)
            closed = _closing(text, opened)
            if name not in ("__launch_bounds__", "__cluster_dims__"):
                break
            at = closed + 1
        body = text.find("{", closed)
        if body >= 0 and not text[closed + 1:body].strip():
            yield name, text[opened:closed + 1], text[body:_closing(text, body, "{}") + 1]


def test_loads_stay_behind_the_wait_for_the_kernel_before():
    """A kernel that waits for the kernel before it (pdl_wait) promises for no pointer but a weight's that nothing else
    writes what it names: loads under such a promise are not ordered behind the wait."""
    waiting, broken = 0, []
    for file in sorted(os.listdir(KERNELS)):
        if not file.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(KERNELS, file)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for name, parameters, body in _kernels(text):
            if "pdl_wait()" not in body:
                continue
            waiting += 1
            broken += [f"{file}: {name}: {p}" for p in re.findall(r"__restrict__\s+(\w+)", parameters) if p not in WEIGHTS]
            broken += [f"{file}: {name}: {x}" for x in re.findall(r"__ldg\(([^;]*)", body) if "bias" not in x]
            broken += [f"{file}: {name}: ld.global.nc" for _ in re.findall(r"ld\.global\.nc", body)]
    assert waiting > 50                      # the sources were found and understood
    assert not broken, broken


def _loops(text):
    """(line, head, body) of every for and while loop; the body of a loop without braces is its statement."""
    for found in re.finditer(r"\b(?:for|while)\s*\(", text):
        closed = _closing(text, found.end() - 1)
        at = closed + 1 + len(text[closed + 1:]) - len(text[closed + 1:].lstrip())
        end = _closing(text, at, "{}") if text[at] == "{" else text.index(";", at)
        yield text.count("\n", 0, found.start()) + 1, text[found.start():closed + 1], text[at:end + 1]


def test_no_warp_waits_for_one_that_gave_up():
    """A bounded wait that runs out in one thread may be completed in the next: a loop that is left after such a wait has nothing in it
    that several warps take part in, and what a warp's lanes take part in only where the lanes agree on the wait."""
    found, broken = 0, []
    for file in sorted(os.listdir(KERNELS)):
        if not file.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(KERNELS, file)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for line, head, body in _loops(text):
            waits = re.findall(r"\bmbar_wait\w*", body)
            left = re.search(r"\bok\b", head) or re.search(r"if \(!(?:ok|mbar_wait\w*\([^;]*)\)\s*(?:break|return)", body)
            if not waits or not left:
                continue
            found += 1
            if re.search(r"bar\.sync|__syncthreads|cluster_sync|barrier\.cluster", body):
                broken.append(f"{file}:{line}: a barrier of several warps")
            if re.search(r"__syncwarp|\w+_sync\(|\btmem_(?:ld|st)", body) and "mbar_wait" in waits:
                broken.append(f"{file}:{line}: lanes that do not agree")
    assert found > 10
    assert not broken, broken
