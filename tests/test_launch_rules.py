"""What launch.cuh asks of a kernel that is scheduled before the launch ahead of it has ended, read from the sources: a
kernel that broke it would fail on a GPU only now and then."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparsetir_b200", "csrc")


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _functions():
    """Every function of the CUDA sources: (file, name, parameters, body), comments taken out."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"\b(\w+)\(", text):
            end = _closing(text, m.end() - 1, "()")
            after = re.match(r"\s*(const\s*)?\{", text[end + 1:])
            if not after or m.group(1) in ("if", "for", "while", "switch"):
                continue
            at = end + after.end()
            found.append((name, m.group(1), text[m.end():end], text[at:_closing(text, at, "{}") + 1]))
    return found


FUNCTIONS = _functions()
LAUNCHED = sorted({m for f in os.listdir(CSRC) if f.endswith(".cu") and f != "launch.cuh"
                   for m in re.findall(r"launch_chained(?:_if)?\([^;]*?\b(\w+_kernel)\b", open(os.path.join(CSRC, f)).read())})


def _kernel(name):
    found = [f for f in FUNCTIONS if f[1] == name]
    assert len(found) == 1, name
    return found[0]


def _reached(kernel):
    """The kernel and what it calls, by name, of its own file and the headers."""
    todo, seen = [_kernel(kernel)], []
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.append(f)
        called = set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", f[3]))
        todo += [g for g in FUNCTIONS if g[1] in called and (g[0] == seen[0][0] or g[0].endswith(".cuh"))]
    return seen


def test_the_chained_kernels_are_found():
    assert {"csrmm_lean_kernel", "csr_split_kernel", "hyb_spmm_lean_kernel", "sddmm_kernel", "sparse_softmax_kernel",
            "bsrmm_persist_kernel", "rgms_tma_kernel", "rgms_f16_tc_kernel", "sparse_conv_kernel",
            "tcspmm_mma_kernel"} <= set(LAUNCHED)


@pytest.mark.parametrize("kernel", LAUNCHED)
def test_operands_are_read_behind_the_wait(kernel):
    """No load that may be moved ahead of the wait: neither __ldg nor ld.global.nc, nor a const __restrict__ pointer, of
    which the compiler makes the same."""
    reached = _reached(kernel)
    assert re.search(r"\bchain_(wait|enter)\(", reached[0][3]), f"{kernel} does not wait"
    for file, name, params, body in reached:
        for what in (r"__ldg\w*\(", r"ld\.global\.nc", r"const [\w:<>\s]+\*\s*__restrict__"):
            assert not re.search(what, params + body), f"{file}: {name}, which {kernel} calls, has {what}"


def test_tensor_memory_is_taken_before_the_next_launch_may_take_it():
    """A block of the next launch takes its tensor memory and then waits for this launch to end: every block of this one
    has to have its own by then."""
    with_tmem = [k for k in LAUNCHED if "tmem_alloc(" in _kernel(k)[3]]
    assert len(with_tmem) >= 5
    for kernel in with_tmem:
        body = _kernel(kernel)[3]
        taken = body.index("__syncthreads()", body.index("tmem_alloc("))  # the block has it behind this barrier
        early = body.find("chain_enter("), body.find("chain_trigger(")
        assert all(at < 0 or at > taken for at in early), kernel


@pytest.mark.parametrize("kernel", LAUNCHED)
def test_every_block_waits_or_has_seen_a_flag(kernel):
    """The first thing that touches memory is the wait, or the flag of a launch that has waited."""
    body = _kernel(kernel)[3]
    waits = [m.start() for m in re.finditer(r"\bchain_(?:wait|enter)\(", body)]
    read = body.find("ld_global(")
    assert read < 0 or waits[0] < read, f"{kernel} reads before it waits"
    depth = lambda at: body.count("{", 0, at) - body.count("}", 0, at)  # noqa: E731
    statement = lambda at: body[max(body.rfind(c, 0, at) for c in ";{}") + 1:at].strip()  # noqa: E731
    plain = [at for at in waits if depth(at) == 1 and statement(at) == ""]
    flagged = [at for at in waits if depth(at) == 1 and re.fullmatch(r"if \(\w+ == nullptr \|\| ld_acquire\(\w+\) == 0\)", statement(at))]
    assert plain or flagged, f"{kernel} waits only under a condition"
    if not plain:  # then one block has to wait before the launch ends
        assert any(depth(at) > 1 and statement(at) == "" for at in waits), kernel
