"""Loads of the kernels that run as programmatic dependents, read from their
sources: such a kernel is resident while the one before it still writes what it
reads, so it may not load that through the non-coherent path (ld.global.nc,
__ldg, const __restrict__ parameters), and an assembly load has to be volatile
with a memory clobber, or the compiler may move it above griddepcontrol.wait."""

from __future__ import annotations

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opendynamo_b200", "csrc")
# read-only while a step runs: what the host or a kernel of an earlier, completed
# call wrote (ensemble layout; the training pools and their row numbers)
READ_ONLY = {"boxes", "tile_map", "Tp", "Xp", "rows"}


def _sources():
    files = [f for p in ("*.cu", "*.cuh", "*.h") for f in glob.glob(os.path.join(CSRC, p))]
    assert len(files) > 10
    return {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(files)}


def _balanced(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced")


def test_assembly_memory_accesses_are_ordered():
    seen = 0
    for name, text in _sources().items():
        for m in re.finditer(r"\basm(\s+volatile)?\s*\(", text):
            body = _balanced(text, m.end() - 1, "()")
            if not re.search(r"\b(ld|st|red|atom)\.(global|shared)|ldmatrix|cp\.async|griddepcontrol", body):
                continue
            seen += 1
            assert m.group(1), f"{name}: {body} is not volatile"
            assert '"memory"' in body, f"{name}: {body} has no memory clobber"
            assert ".nc" not in body, f"{name}: {body} is non-coherent"
    assert seen > 10


def _dependent_kernels():
    for name, text in _sources().items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*)?", text):
            i = m.end()
            if text[i] == "(":
                i += len(_balanced(text, i, "()"))
            k = re.compile(r"\s*(\w+)\s*").match(text, i)
            params = _balanced(text, k.end(), "()")
            body = _balanced(text, text.index("{", k.end() + len(params)), "{}")
            if "dependent_start()" in body or "griddepcontrol.wait" in body:
                yield name, k.group(1), params, body


def test_dependent_kernels_read_coherently():
    found = {k: (params, body) for _, k, params, body in _dependent_kernels()}
    assert {"stage_a_kernel", "stage_b_split_kernel", "ensemble_a_kernel", "ensemble_b_kernel", "gather_kernel",
            "loss_grad_kernel", "grad_finish_kernel", "adam_kernel", "mlp_fused_kernel"} <= set(found)
    for kernel, (params, body) in found.items():
        assert "__ldg" not in body, kernel
        for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
            assert p in READ_ONLY, f"{kernel}: {p}"


@pytest.mark.parametrize("name", ["od_stage.cuh", "od_mlp.cuh", "od_mlp_fused.cuh", "od_ensemble.cu"])
def test_their_device_functions_read_coherently(name):
    """(Files whose device functions run in such kernels.)"""
    assert "__ldg" not in _sources()[name]


def test_row_sums_read_coherently():
    text = _sources()["od_closure.cu"]
    i = text.index("float row_sum(")
    assert "__ldg" not in _balanced(text, text.index("{", i), "{}")


def test_weights_are_complete_when_the_call_that_writes_them_returns():
    """(The inference kernel reads them before griddepcontrol.wait.)"""
    text = _sources()["od_closure.cu"]
    writers = set()
    for m in re.finditer(r"\bint (od_mlp_\w+)\(", text):
        params = _balanced(text, m.end() - 1, "()")
        i = m.end() - 1 + len(params)
        if text[i:i + 2] == ";\n":
            continue
        body = _balanced(text, text.index("{", i), "{}")
        if re.search(r"cast_weights_kernel|adam_kernel|tile_fused_weights|cudaMemcpyAsync\(m->w\b", body):
            writers.add(m.group(1))
            last = max(body.rfind("cudaStreamSynchronize(m->stream)"), body.rfind("read_status(m"))
            assert last > max(body.rfind(k) for k in ("cast_weights_kernel", "adam_kernel", "tile_fused_weights")), m.group(1)
    assert writers == {"od_mlp_set_params", "od_mlp_train_step"}
