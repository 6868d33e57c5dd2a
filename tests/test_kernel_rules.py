"""Rules that the kernels' text has to keep because a run on a GPU shows a break only by chance."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama2.jl_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def closing(text, at):
    """Index of the bracket that closes the one at `at`."""
    pairs = {"(": ")", "{": "}"}
    opened, closed, depth = text[at], pairs[text[at]], 0
    for i in range(at, len(text)):
        depth += (text[i] == opened) - (text[i] == closed)
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        end = closing(text, m.end() - 1)
        start = text.index("{", end)
        yield m.group(1), text[m.end():end], text[start:closing(text, start) + 1]


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh"))

# What the kernels of a file read through the read-only path: weights, gains, biases, tables, and index lists that the host
# uploaded before the chain of launches began.
CONSTANTS = {
    "attention.cuh": {"p.pos_list"},
    "dense_gemm.cuh": {"e.bias"},
    "dense_matvec.cuh": {"p.upd.w", "p.upd.step"},
    "dense_ops.cuh": {"cs", "e.bias", "e.tokens", "n.w", "n.b"},
    "fused_matvec.cuh": {"p.gain", "p.rope_cs", "d6A", "d6B", "wa", "wb"},
    "head_attention.cuh": {"w", "cs"},
    "kq_gemm.cuh": {"s", "sg.d6"},  # s: the gains
    "latent_attention.cuh": {"p.dnorm", "p.sink"},
    "latent_prefill.cuh": {"p.sink"},
    "mlstm.cuh": {"p.norm"},
    "mlstm_prefill.cuh": {"p.m.norm"},
    "prefill_ops.cuh": {"tokens", "p.pos_list", "p.rope_cs"},
    "stack_rows.cuh": {"tv", "pv", "p.index", "p.upd.w", "p.upd.step"},
    "token_kernel.cuh": {"s4", "tp.ops", "d6A", "d6B"},
}


@pytest.mark.parametrize("name", FILES)
def test_read_only_path_for_constants(name):
    """Kernels start while their predecessor still writes, and the read-only path (__ldg, const __restrict__) is defined only for memory that nobody
    writes while the kernel runs: such a load may be moved above the wait, and its line may be an old one."""
    text = source(name)
    for m in re.finditer(r"\b__ldg\(", text):
        arg = text[m.end():closing(text, m.end() - 1)]
        arg = re.sub(r"reinterpret_cast<[^>]*>\(", "", arg).lstrip("&(")
        root = re.match(r"[\w.]*\w", arg).group(0)
        assert root in CONSTANTS.get(name, set()), f"{name}: __ldg({arg})"
    for kernel, params, body in kernels(text):
        if "pdl_wait()" in body:
            inputs = set(re.findall(r"const [\w:]+\*\s*__restrict__\s+(\w+)", params))
            assert inputs <= {"table", "d6", "rope"}, f"{name}: {kernel}"


BARRIER = re.compile(r"bar\.sync|\bpa_bar_sync\(|\bpartial_sync(?:_2)?\(|\bconsumer_sync\(|\bblock_sum(?:_all)?\b")


def loops(text):
    """Body of every loop with braces."""
    for m in re.finditer(r"\bfor\s*\(|\bwhile\s*\(", text):
        end = closing(text, m.end() - 1)
        start = re.match(r"\s*(?:for\s*\([^{]*\)\s*)?", text[end + 1:]).end() + end + 1  # (two headers over one body)
        if text[start] == "{":
            yield text[start:closing(text, start) + 1]


def conditions(text):
    """(condition, what is done) of every if with braces."""
    for m in re.finditer(r"\bif\s*\(", text):
        end = closing(text, m.end() - 1)
        start = re.match(r"\s*", text[end + 1:]).end() + end + 1
        stop = closing(text, start) + 1 if text[start] == "{" else text.index(";", start) + 1
        yield text[m.end():end], text[start:stop]


@pytest.mark.parametrize("name", FILES)
def test_no_warp_leaves_a_loop_with_a_barrier(name):
    """A bounded wait may run out for one warp and not for the next.  Where warps meet at a named barrier, which has no bound, the verdict is carried along
    to the loop's end: a warp that left would be waited for without end."""
    for kernel, _, body in kernels(source(name)):
        for loop in loops(body):
            if BARRIER.search(loop):
                for cond, then in conditions(loop):
                    assert not ("mbar_wait" in cond and re.search(r"\b(break|return)\b", then)), f"{name}: {kernel}: {cond}"


def headers(text, at):
    """What stands in front of every brace that is open at `at`."""
    out, depth = [], 0
    for i in range(at - 1, -1, -1):
        depth += (text[i] == "}") - (text[i] == "{")
        if depth < 0:
            depth = 0
            out.append(text[max(text.rfind(c, 0, i) for c in ";{}") + 1:i])
    return out


@pytest.mark.parametrize("name", [f for f in FILES if "tmem_ld" in source(f) and f != "tcgen05.cuh"])
def test_a_warp_decides_together_whether_a_wait_ran_out(name):
    """Loads and stores of tensor memory, votes and shuffles need all threads of a warp.  So where a whole warp waits, its threads agree on the verdict; alone
    wait only threads that work alone."""
    for kernel, _, body in kernels(source(name)):
        for m in re.finditer(r"\bmbar_wait_(?:bounded|parked)\(", body):
            together = re.search(r"__all_sync\(0xffffffffu,\s*$", body[:m.start()])
            assert together or any("lane == 0" in h for h in headers(body, m.start())), f"{name}: {kernel}: {body[m.start():m.start() + 60]}"
