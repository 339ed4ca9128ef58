"""Orders inside the kernels that no run shows reliably, read from their sources."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "speed3r_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def kernels_with_tensor_memory():
    found = []
    for path in SOURCES:
        if os.path.basename(path) == "common.cuh":
            continue
        for m in re.finditer(r"\btmem_alloc\(", code(path)):
            found.append(pytest.param(path, m.start(), id=os.path.basename(path)))
    return found


@pytest.mark.parametrize("path, at", kernels_with_tensor_memory())
def test_next_kernel_starts_after_tensor_memory_is_allocated(path, at):
    """A CTA of the next kernel that allocates first waits for this kernel's end with the columns this CTA waits for.  The
    trigger comes after a barrier behind the allocation."""
    src = code(path)
    start = src.rfind("\n}", 0, at)                    # the function before
    body = src[start:src.find("\n}", at)]
    at -= start
    launch = body.find("griddep_launch()")
    barrier = body.find("__syncthreads()", at)
    assert 0 <= barrier < launch, "griddep_launch() before the barrier behind tcgen05.alloc"


def functions_that_order_launches():
    found = []
    for path in SOURCES:
        if os.path.basename(path) == "common.cuh":
            continue
        for body in code(path).split("\n}"):
            if "griddep_" in body:
                name = re.findall(r"\b(\w+)\(", body[body.index("__device__" if "__device__" in body else "__global__"):])
                name = [n for n in name if n != "__launch_bounds__"][0]
                found.append(pytest.param(body, id=f"{os.path.basename(path)}:{name}"))
    return found


@pytest.mark.parametrize("body", functions_that_order_launches())
def test_what_other_kernels_wrote_is_read_behind_the_wait_for_them(body):
    """griddepcontrol.wait is all that makes the writes of the kernels in front visible: every thread goes through it, once, before it reads
    global memory and before it lets the next kernel start."""
    assert body.count("griddep_wait(") == 1 and body.count("griddep_launch(") == 1
    wait = re.search(r"\n  griddep_wait\(\);", body)
    assert wait, "the wait is not for every thread"
    before = body[:wait.start()]
    assert "griddep_launch(" not in before
    assert not re.search(r"\b(tma_load|__ldg|ldg_|cp_async|wait_bound|ld\.(relaxed|acquire|global)|prefetch)", before)


@pytest.mark.parametrize("path", sorted({p.values[0] for p in kernels_with_tensor_memory()}), ids=os.path.basename)
def test_draining_after_a_wait_that_gave_up_signals_no_result(path):
    """The issuing warp commits once more after a wait that gave up, to see its products drained.  The barrier of that commit is not one
    that tells other warps their results are there: they may have got past their own waits, and would store what is not finished."""
    src = code(path)
    committed = set(re.findall(r"umma_commit\([^;]*?&ctl\.(\w+)", src)) | set(re.findall(r"umma_commit\([^;]*:\s*&ctl\.(\w+)", src))
    drains = set(re.findall(r"\bmbar_wait\(&ctl\.(\w+)[^;]*&dummy\)", src)) & committed
    waited = set(re.findall(r"mbar_wait_warp\(&ctl\.(\w+)[^;]*?abort_flag\)", src))
    assert drains and not drains & waited, f"{os.path.basename(path)}: {drains & waited}"


def test_a_rows_two_threads_do_not_overwrite_what_they_tell_each_other():
    """End of the collection: a row's two threads exchange words between meetings, the only thing that orders them.  A word that one of
    them reads between two meetings is written in front of the first or behind the second."""
    src = code(os.path.join(CSRC, "cmp_topk.cuh"))
    src = src[src.index("uint32_t* tell = words"):]
    src = src[src.index(";") + 1:]

    def words_of(index):
        if "par" in index:                     # either thread's own or the other's largest key
            return {0, 1}
        return {eval(index) // 128}

    phases, seen = src.split("meet();"), set()
    assert len(phases) == 4
    for n, phase in enumerate(phases):
        written, read = set(), set()
        for m in re.finditer(r"\btell\[([^\]]*)\](\s*=(?!=))?", phase):
            (written if m.group(2) else read).update(words_of(m.group(1)))
        assert not written & read, f"words {written & read} between meetings {n} and {n + 1}"
        assert read <= seen
        seen |= written


def test_polynomial_exponential_is_as_exact_as_stated():
    """2^f on [-1/2, 1/2] with the coefficients of exp2_fma2, in 64 bits and with every step rounded to fp32."""
    import numpy as np
    src = open(os.path.join(CSRC, "common.cuh")).read()
    body = src[src.index("float2 exp2_fma2(float2 x)"):]
    body = body[:body.index("\n}")]
    coeff = [np.float32(c) for c in re.findall(r"make_float2\(([0-9.e+-]+)f, \1f\)", body)][2:]      # behind the two shifts
    assert len(coeff) == 6 and coeff[-1] == 1
    f = np.linspace(-0.5, 0.5, 200001).astype(np.float32).astype(np.float64)
    exact = r = np.zeros_like(f)
    for c in coeff:
        exact = exact * f + np.float64(c)
        r = (r * f + np.float64(c)).astype(np.float32).astype(np.float64)
    assert np.abs(exact / 2.0 ** f - 1).max() < 1.65e-7
    assert np.abs(r / 2.0 ** f - 1).max() < 2.25e-7


def test_shared_memory_limits_do_not_depend_on_the_call():
    """cudaFuncSetAttribute changes a kernel for every thread of the process: the limit is a constant, or the largest of all."""
    for path in SOURCES:
        for limit in re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)\)?;", code(path), flags=re.S):
            names = set(re.findall(r"[A-Za-z_]\w*", limit)) - {"static_cast", "int", "sizeof", "int32_t"}
            assert all(re.match(r"k[A-Z]|C$|AtCfg|TkCfg|R$", n) for n in names), f"{os.path.basename(path)}: {limit}"
