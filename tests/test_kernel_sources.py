"""Rules of programmatic dependent launch that the kernels' sources keep (csrc/common.cuh states them): read as text, so that
they hold for every size and build, where a run shows a fault only when its timing happens to be bad."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "odin_infer_b200", "csrc")
SOURCES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# what no kernel of a step writes: weights, constant tables, the step's integer tables
CONSTANT = {"w", "W", "table", "pair", "bias", "cos_t", "sin_t", "sink", "mu", "params", "in_bias", "y_bias", "log_decay", "decay",
            "tok_pos", "tok_seq", "block_table", "seq_start", "seq_slots", "rows"}


def _without_comments(text):
    text = re.sub(r"//[^\n]*", "", text)
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def _block(text, at):
    """From the opening brace at `at` to its closing one."""
    depth, i = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[at:i]


def _functions(name):
    """(name, parameters, body) of every device function of a source that waits for the kernel before it or allocates tensor memory."""
    with open(os.path.join(CSRC, name)) as f:
        text = _without_comments(f.read())
    for m in re.finditer(r"\b(\w+)\s*\(((?:[^(){};]|\([^(){};]*\))*)\)\s*\{", text):
        if m.group(1) in ("if", "for", "while", "switch") or not re.search(r"__(global|device)__[^;{}]*$", text[:m.start()]):
            continue
        body = _block(text, m.end() - 1)
        if "pdl_wait()" in body or "tmem_alloc" in body:
            yield m.group(1), m.group(2), body


def _reads_ahead(params, body):
    before = body[:body.index("pdl_wait()")]
    pointers = re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)", params) + re.findall(r"VecRef\s+(\w+)", params)
    return bool(re.search(r"^\s*(fetch|load_w|load)\(", before, flags=re.M)) or any(
        re.search(r"\b%s\s*(\[|\.at4?\()|\b(ld4|load4w?(<\w+>)?)\(%s\b|\*>\(%s \+" % (p, p, p), before) for p in pointers)


@pytest.mark.parametrize("source", SOURCES)
def test_what_earlier_kernels_write_is_not_read_as_invariant(source):
    """A load through `const T* __restrict__` counts as invariant and may be moved ahead of the wait for the kernel that writes
    what it reads; kernels that read anything ahead of the wait take such inputs through plain pointers."""
    for name, params, body in _functions(source):
        if "pdl_wait()" not in body or not _reads_ahead(params, body):
            continue
        invariant = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)) - CONSTANT
        assert not invariant, (source, name, sorted(invariant))


@pytest.mark.parametrize("source", SOURCES)
def test_tensor_memory_is_held_before_the_next_kernel_may_start(source):
    """A kernel that allows the next launch and allocates afterwards can wait for columns that a later kernel holds, which waits
    for this one to end."""
    for name, params, body in _functions(source):
        if "pdl_trigger()" in body and "tmem_alloc" in body:
            assert body.index("tmem_alloc") < body.index("pdl_trigger()"), (source, name)


@pytest.mark.parametrize("source", SOURCES)
def test_no_wait_for_either_phase(source):
    """One of a barrier's two parities always counts as complete: a wait for the one or the other waits for nothing."""
    with open(os.path.join(CSRC, source)) as f:
        text = _without_comments(f.read())
    for bar in re.findall(r"try_wait\(([^;]*?), [01]\) \|\|", text):
        assert f"try_wait({bar}, 0) || tc::mbar_try_wait({bar}, 1)" not in text, (source, bar)


@pytest.mark.parametrize("source", SOURCES)
def test_shared_memory_limits_only_grow(source):
    """A kernel's limit belongs to all threads: with sizes of single calls it is set where it cannot be lowered (odin_allow_smem)."""
    with open(os.path.join(CSRC, source)) as f:
        text = _without_comments(f.read())
    if source == "common.cuh":
        text = text.replace(_block(text, text.index("{", text.index("odin_allow_smem"))), "")
    for size in re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*)\)", text):
        assert not re.search(r"\(int\)\s*(smem|bytes|co_smem)\b", size), (source, size)

