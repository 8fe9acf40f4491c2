"""The rules that make programmatic dependent launch sound, read off the kernels' source: a kernel waits before it
triggers and before it leaves, so that it runs beside its direct predecessor only; it reads the solve's status behind
the wait; one whose vectors the next kernel reads through the read-only path triggers after it has written them."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "if-dda_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def _kernels():
    """(name, body) of every kernel that is launched early."""
    for text in SOURCES.values():
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^{;]*?\) )?(k_\w+)\([^{;]*\) \{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            if "pdl_wait()" in text[m.end():i]:
                yield pytest.param(text[m.end():i], id=m.group(1))


KERNELS = list(_kernels())


def test_the_early_launched_kernels_are_found():
    assert {k.id for k in KERNELS} == {"k_fwd_x", "k_pass_y", "k_zconv", "k_inv_x", "k_vec"}


@pytest.mark.parametrize("body", KERNELS)
def test_waits_before_trigger_and_exit(body):
    for m in re.finditer(r"\breturn\b|pdl_trigger\(\)", body):
        assert "pdl_wait()" in body[:m.start()], body[max(0, m.start() - 80):m.end()]


@pytest.mark.parametrize("body", [k for k in KERNELS if k.id in ("k_inv_x", "k_vec")])
def test_triggers_after_its_vectors_are_written(body):
    trigger = body.index("pdl_trigger()")
    last_write = max(body.rfind(w) for w in ("x_load_pairs", "InvXStore", "op.elem"))
    assert 0 < last_write < trigger
    assert re.search(r"__syncthreads\(\);\s*$", body[:trigger])  # every thread's, not the first one's alone


@pytest.mark.parametrize("body", KERNELS)
def test_a_finished_solve_returns_behind_the_wait(body):
    # the branch also keeps read-only loads, which the compiler may move across the wait itself, behind it
    tail = body[body.rindex("pdl_wait();"):]
    assert re.match(r"pdl_wait\(\);\s*(pdl_trigger\(\);\s*)?if \((a\.status && a\.)?status\[rhs\]\) (return;|\{)", tail)
    assert "status" not in body[:body.rindex("pdl_wait();")]


def test_read_only_loads():
    # tables and polarisabilities, which do not change during a solve, or vectors that are written before the trigger
    for arg in re.findall(r"__ldg\((\w+(?:\.\w+)?)", SOURCES["matvec_kernels.cuh"]):
        assert arg in ("tab", "alpha", "dst.tab", "x", "bv"), arg
