"""Kernels that may be started while the kernel before them still writes their
inputs (csrc/common.cuh, after_previous) read those by ordinary loads: a
const __restrict__ parameter and ld.global.nc (__ldg) promise that nothing writes
the memory while the kernel exists, so that the load may come before the wait."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "nerf-tf2_gb300" / "csrc"


def _kernels(text):
    """(name, parameters, body) of the file's __global__ functions."""
    for m in re.finditer(r"__global__ void\s*(?:__launch_bounds__\([^;{]*?\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        parameters, depth, j = text[m.end():i - 1], 1, text.index("{", i) + 1
        start = j
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), parameters, text[start:j]


def test_inputs_of_early_launches_are_ordinary_loads():
    found = set()
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for name, parameters, body in _kernels(text):
            if "after_previous()" not in body:
                continue
            found.add(name)
            inputs = [p.strip() for p in parameters.split(",") if re.match(r"\s*const\b.*\*", p)]
            assert inputs and not [p for p in inputs if "__restrict__" in p], (name, inputs)
            assert "__ldg" not in text and "ld.global.nc" not in text, path.name
            # the wait comes before anything that could read
            before = body[:body.index("after_previous()")]
            assert not re.search(r"\w\s*\[[^\]]*\]\s*[;=)]", before.replace("smem[]", "")), (name, before)
    assert found == {"coarse_sample_kernel", "composite_kernel", "fine_sample_kernel", "mlp_tc_kernel"}, found


def test_every_early_launch_is_of_such_a_kernel():
    launched = set()
    for path in sorted(CSRC.glob("*.cu")):
        launched |= set(re.findall(r"launch_after\((\w+),", path.read_text()))
    assert launched == {"coarse_sample_kernel", "composite_kernel", "fine_sample_kernel"}, launched
