"""Kernels launched as programmatic dependents (they wait for their predecessors themselves) read what an earlier kernel
wrote by plain loads: the read-only path (__ldg, ld.global.nc, a const __restrict__ kernel parameter) is defined only for
data that nothing writes while the kernel lives, and such a kernel's life begins before its predecessors' writes. Checked on
the sources: that path is for weights, codebooks and biases alone."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "c0ven_b200" / "csrc"
CONSTANT_PARAMS = {"W", "bias", "gate", "grid_global"}  # the router's rows, its bias, its gate vector, the codebooks
CONSTANT_ROOTS = {"s", "sc", "w", "wp", "q", "qs", "ql", "qh", "quants_at", "a.grid", "a.w_unscale"}  # pieces of weight matrices and tables
READ_ONLY = re.compile(r"\b(?:__ldg|ldg16|ldg_stream16|ldg_stream8)\(")


def closing(text, at, pair):
    """The place after the bracket that closes the one at text[at]."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def kernels(text):
    """(start, end, name, parameters, body) of every __global__ function's definition."""
    for m in re.finditer(r"\b__global__\b", text):
        n = re.compile(r"\b(k_\w+)\(").search(text, m.end())
        p1 = closing(text, n.end() - 1, "()")
        b0 = text.index("{", p1)
        if ";" in text[p1:b0]:
            continue  # a declaration
        b1 = closing(text, b0, "{}")
        yield m.start(), b1, n.group(1), text[n.end():p1 - 1], text[b0:b1]


def root(argument):
    """The name a load's address starts from, casts and brackets taken off."""
    argument = re.sub(r"\(const [\w ]+\*\)", "", argument)
    return re.match(r"[(\s]*([A-Za-z_]\w*(?:\.\w+)?)", argument.replace("Dec::", "")).group(1)


def test_dependents_read_the_steps_data_by_plain_loads():
    dependents, loads = 0, 0
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for start, end, name, params, body in reversed(list(kernels(text))):
            if "wait_for_predecessors" not in body:
                text = text[:start] + text[end:]  # launched the ordinary way: nothing else runs while it does
                continue
            dependents += 1
            read_only = {p.split()[-1].lstrip("*") for p in params.split(",") if "const " in p and "__restrict__" in p}
            assert read_only <= CONSTANT_PARAMS, (path.name, name, read_only - CONSTANT_PARAMS)
        for m in READ_ONLY.finditer(text):
            argument = text[m.end():closing(text, m.end() - 1, "()") - 1]
            if argument.startswith("const void"):
                continue  # the helper's own definition
            loads += 1
            assert root(argument) in CONSTANT_ROOTS, (path.name, argument)
    assert dependents >= 14 and loads >= 60  # the pattern still finds them


def test_the_check_sees_a_load_that_breaks_the_rule():
    assert root("(const int4 *)(a.act.q + row * a.act.q_stride) + c") == "a.act"
    assert root("a.ngroups") == "a.ngroups" and root("places + k") == "places"
    (_, _, name, params, body), = kernels("static __global__ void __launch_bounds__(256) k_x(const int *__restrict__ ids, int n) { if (n) { f(); } }")
    assert name == "k_x" and "__restrict__ ids" in params and body.count("{") == 2
