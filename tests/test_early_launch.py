"""CPU checks of the sources of the kernels that are launched early (launch.cuh): such a kernel may be
resident while the kernel before it still writes, so it waits before it reads, and it reads what another
kernel writes by loads that may neither move above the wait nor go past the coherent path."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "hermite-teno_gb300" / "csrc"
# __restrict__ parameters that need no after_wait: memory that no kernel writes while its readers may be
# resident, and memory that the kernel only writes (after the wait)
EXEMPT = {"k_batch_stage": {"inst", "jobs"}, "k_train": {"X", "Y", "Gp", "Lp", "err"}}


def sources():
    out = {}
    for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        out[p.name] = re.sub(r"//[^\n]*", "", p.read_text())
    return out


def braced(text, at):
    """The text from the first brace at or after `at` to its partner."""
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def kernel(src, name):
    """Parameter list and body of the kernel `name`."""
    for text in src.values():
        m = re.search(r"__global__[^;{]*\b" + name + r"\s*\(", text)
        if m:
            body = braced(text, m.end())
            return text[m.end():text.index("{", m.end())], body
    raise AssertionError(name)


def early_kernels(src):
    names = set()
    for text in src.values():
        names |= set(re.findall(r"launch_early\(\s*[^,]+,\s*(k_\w+)", text))
    return sorted(names)


def test_early_kernels_wait_and_read_coherently():
    src = sources()
    names = early_kernels(src)
    assert {"k_begin_step", "k_end_step", "k_fused", "k_batch_stage", "k_adam", "k_train"} <= set(names)
    for name in names:
        params, body = kernel(src, name)
        assert "grid_wait();" in body, name
        after = body.split("grid_wait();", 1)[1]
        assert "__ldg(" not in body and "ld.global.nc" not in body, name
        for p in re.findall(r"__restrict__\s+(\w+)", params):
            assert p in EXEMPT.get(name, ()) or f"{p} = after_wait({p})" in after, (name, p)


def test_early_stage_reads_its_state_after_the_wait():
    """The mixed FV 2D stage: the state that the stage before it writes."""
    src = sources()
    tile = braced(src["fv2d_fused.cuh"], src["fv2d_fused.cuh"].index("double tile_stage("))
    assert "__ldg(" not in tile
    args = braced(src["fv2d_fused.cuh"], src["fv2d_fused.cuh"].index("struct StageArgs"))
    assert "__restrict__" not in args and "__restrict__" not in tile
    # the ghost cells' loads go through a parameter without __restrict__
    ghost = src["fv2d_common.cuh"]
    head = ghost[ghost.index("void bc_state("):]
    assert "__restrict__" not in head[:head.index("{")]


def test_train_reads_the_callers_rows_only_behind_a_full_dependency():
    """k_train fetches its first rows before grid_wait.  The kernel before an epoch's first batch may be
    the caller's that wrote them, so that batch is not launched early; the later ones follow k_adam,
    which does not write rows."""
    text = sources()["mlp.cu"]
    early = re.findall(r"launch_early\(\s*([^,]+),\s*k_train\b", text)
    assert early == ["off > 0"]
    _, body = kernel({"mlp.cu": text}, "k_adam")
    assert not re.search(r"\b[XY]\b", body)
