"""Kernels that may start while the kernel before them still writes (launched
through launch_chained with its first argument not false) must not read what
that kernel writes through the read-only path: ld.global.nc is defined only for
memory that nothing writes during the reading kernel's whole life, and the
compiler may move such a load above the wait.  This reads the sources: in those
kernels, and in every device function they reach, __ldg is applied to the
constant tables (twiddles, Poseidon2 tables) only.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pico_b200" / "csrc"
# what __ldg may read in a chained kernel: twiddle tables, and the field's Poseidon2 tables
CONSTANT = re.compile(r"^(tw\.(lo|hi|stage)\b|src \+ i$)")


def _sources():
    text = "\n".join((CSRC / f).read_text() for f in ("p2_lane.cuh", "p2_tc.cuh", "p2_kernels.cu"))
    return re.sub(r"//[^\n]*", "", text)


def _balanced(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _functions(text):
    """name -> bodies of every function defined in the text."""
    out = {}
    for m in re.finditer(r"\b(\w+)\(", text):
        if m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__", "asm", "volatile"):
            continue
        end = _balanced(text, m.end() - 1, "()")
        tail = re.match(r"\s*(const\s*)?\{", text[end + 1:])
        if not tail:
            continue
        at = end + 1 + tail.end() - 1
        out.setdefault(m.group(1), []).append(text[at:_balanced(text, at, "{}") + 1])
    for m in re.finditer(r"#define (PICO_TC_\w+)\(.*\)((?:.*\\\n)*.*)", text):
        out.setdefault(m.group(1), []).append(m.group(2))
    return out


def _chained_kernels(text):
    names = set()
    for m in re.finditer(r"\b(launch_chained|tc_launch)\(", text):
        call = text[m.end():_balanced(text, m.end() - 1, "()")]
        if not call.startswith("false"):
            names |= set(re.findall(r"\bk_\w+", call))
    return names


def test_chained_kernels_read_only_constants_through_ldg():
    text = _sources()
    functions = _functions(text)
    kernels = _chained_kernels(text)
    assert {"k_subtree_lane", "k_compress_tc", "k_fri_fold_hash_lane", "k_fri_fold_hash_tc",
            "k_challenger_observe"} <= kernels
    todo, reached = list(kernels), set()
    while todo:
        name = todo.pop()
        if name in reached or name not in functions:
            continue
        reached.add(name)
        for body in functions[name]:
            todo += re.findall(r"\b(\w+)(?:<[\w, ]*>)?\(", body)
    assert {"fri_fold_row", "half_beta", "lane_subtree", "lane_load_tables", "open"} <= reached
    bad = []
    for name in sorted(reached):
        for body in functions[name]:
            for m in re.finditer(r"\b__ldg\(", body):
                arg = body[m.end():_balanced(body, m.end() - 1, "()")]
                if not CONSTANT.match(arg):
                    bad.append(f"{name}: __ldg({arg})")
    assert not bad, bad


def test_chained_kernels_wait_for_the_kernel_before_them():
    functions = _functions(_sources())
    for name in _chained_kernels(_sources()):
        for body in functions[name]:
            assert re.search(r"lane_load_tables<F>\(|PICO_TC_OPEN\(", body), name
    for waits in ("lane_load_tables", "open"):
        assert all("grid_wait()" in body for body in functions[waits]), waits


def test_tensor_memory_is_taken_before_a_successor_may_start():
    # a waiting successor holds tensor memory: with its own still to come, a CTA
    # could wait for columns that are given back only after it has finished
    body, = _functions(_sources())["open"]
    taken = body.index("__syncthreads()", body.index("tcgen05.alloc"))
    assert taken < body.index("grid_release()") < body.index("grid_wait()")
