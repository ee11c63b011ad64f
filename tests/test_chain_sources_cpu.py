"""Kernels launched by programmatic dependence (launch_chained) begin while the kernel before them still writes.  What they
may then do is a matter of their source, which this looks at; a wrong order of a load would show as a wrong value at best
once in a while."""
import os
import re

import pytest

from moe_gen_b200 import build as b

# operands that are complete before the first kernel of a forward begins: the caller's, and the packed weights
OLDER = {"x", "gate_w", "bias", "w", "weight", "b8"}
# __ldg of: rows of x in the scatter, router operands, weight scales
LDG_OLDER = ("src + v", "xr + v", "wr + v", "reinterpret_cast<const uint2*>(xr[j])", "reinterpret_cast<const uint2*>(w +",
             "srow +", "row + i * 32", "weight + v")


def _strip(text):
    return re.sub(r"//[^\n]*", "", text)


def _functions(files, head):
    """name -> (parameters, body) of every function whose head matches; bodies of one name together"""
    out = {}
    for f in files:
        text = _strip(open(os.path.join(b.CSRC, f)).read())
        for m in re.finditer(head, text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            j = text.index("{", i)
            if ";" in text[i:j]:
                continue                  # declared here, defined elsewhere
            depth, i = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            old = out.get(m.group(1), ("", ""))
            out[m.group(1)] = (old[0] + ", " * bool(old[0]) + params, old[1] + text[j + 1:i - 1])
    return out


KERNELS = _functions(b.SOURCES, r"__global__[^;{]*?(\w+_kernel)\s*\(")
HELPERS = _functions(b.SOURCES + ["common.cuh", "tc.cuh"], r"__device__ __forceinline__ [^;{(]*?(\w+)\s*\(")
CHAINED = sorted(n for n, (_, body) in KERNELS.items() if "chain_wait()" in body)


def test_every_kernel_launched_by_dependence_waits():
    launched = set()
    for f in b.SOURCES:
        text = _strip(open(os.path.join(b.CSRC, f)).read())
        launched |= set(re.findall(r"launch_chained\(\s*h,\s*(\w+)", text))
        if "cudaLaunchAttributeProgrammaticStreamSerialization" in text:
            launched |= set(re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(\w+_kernel)", text))
    assert len(launched) >= 8 and "combine_kernel" in launched
    assert launched == set(CHAINED)


@pytest.mark.parametrize("name", CHAINED)
def test_no_read_only_path_for_what_a_predecessor_writes(name):
    """__ldg, and __restrict__ on a pointer that is only read, promise memory that nothing writes while the kernel lives:
    the load may come from the non-coherent path and may be moved ahead of the wait.  The same for what the kernel calls."""
    todo, seen = [name], {}
    while todo:
        f = todo.pop()
        seen[f] = KERNELS[f] if f in KERNELS else HELPERS[f]
        todo += [g for g in set(re.findall(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\(", seen[f][1])) if g in HELPERS and g not in seen]
    for f, (params, body) in seen.items():
        for p in params.split(","):
            if "__restrict__" in p:
                assert p.split()[-1] in OLDER, f"{f}: {p.strip()}"
        for m in re.finditer(r"__ldg\(", body):
            assert body[m.end():].startswith(LDG_OLDER), f"{f}: __ldg({body[m.end():m.end() + 40]}"
    assert "copy_row" in seen or name not in ("permute_rows_kernel", "plan_small_kernel")


@pytest.mark.parametrize("name", CHAINED)
def test_every_thread_waits_before_it_reads_memory(name):
    """What a predecessor has written is visible to a thread behind its own wait; the begin of a kernel promises nothing,
    about older kernels either.  A value may be peeked at before, as a guess, if it is read again behind the wait."""
    params, body = KERNELS[name]
    at = body.index("chain_wait()")
    before, behind = body[:at], body[at:]
    for m in re.findall(r"\bpeek\(([\w.]+)", before):
        assert m in behind, f"{name}: {m} is only guessed"
    assert "peek(" not in behind
    before = re.sub(r"\bpeek\([\w.]+", "peek(", before)
    assert before.count("{") == before.count("}"), f"{name}: only some threads reach the wait"
    pointers = [p.split()[-1].lstrip("*") for p in params.split(",") if "*" in p]
    used = [p for p in pointers if re.search(rf"\b{p}\b", before)]
    used += re.findall(r"\bg\.(?:pad_offsets|counts|next_job|scales|out)\b", before)
    assert not used, f"{name}: {used} before the wait"


def test_the_plan_that_copies_lets_the_gemm_go_behind_its_counting():
    """Where the plan copies the rows too, the weight-lane GEMM comes straight behind it, begins as soon as every block has let it
    go, and peeks at the counts: the block that stores them lets it go when it has counted, and the peek comes last in the GEMM's
    own preparation, so that it shows this call's counts and not what an earlier call left there."""
    _, body = KERNELS["plan_small_kernel"]
    assert re.findall(r"([^\n;]*)chain_go\(\)", body) == ["  if (!COPY || !stores) ", "  if (COPY && stores) "]
    assert "stores = !COPY || blockIdx.x == 0" in body[:body.index("chain_go()")]
    counted = body[body.index("atomicOr(&bm"):body.rindex("chain_go()")]
    assert "__syncthreads();" in counted and "counts[tid] =" not in counted
    _, body = KERNELS["grouped_gemm_wl_kernel"]
    assert body.index("tcgen05.alloc") < body.index("cluster_sync_all()") < body.index("peek(") < body.index("chain_wait()")
