"""Kernels launched with launch_chained (chain.cuh) are resident while the
kernels before them still store what they will read, so only the caller's
field, complete before the first of them starts, may be read through the
read-only path.  Checked on the sources: no function reachable from a chained
kernel has a `const ... __restrict__` parameter or an __ldg on anything else,
and the kernels that read the field first are launched plainly."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "prism_b200", "csrc")
FIELD = {"data", "base"}  # the field, and a tile's first value in it
FILES = ["autotune.cuh", "bitplane.cuh", "flat.cuh", "predict.cuh", "zbpc.cuh", "prism_b200.cu"]


def _closing(s, at, pair):
    depth = 0
    for i in range(at, len(s)):
        depth += (s[i] == pair[0]) - (s[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _sources():
    text = ""
    for f in FILES:
        with open(os.path.join(CSRC, f)) as fh:
            text += re.sub(r"//[^\n]*", "", fh.read()) + "\n"
    return text


def _functions(text):
    """name -> [(parameters, body)] of the device functions and kernels."""
    out = {}
    for m in re.finditer(r"__(?:device|global)__[\w\s:<>*&,()]*?\b(\w+)\s*\(", text):
        name = m.group(1)
        if name == "__launch_bounds__":  # the name follows its parenthesis
            end = _closing(text, m.end() - 1, "()")
            m2 = re.compile(r"\s*(\w+)\s*\(").match(text, end + 1)
            name, at = m2.group(1), m2.end() - 1
        else:
            at = m.end() - 1
        close = _closing(text, at, "()")
        brace = re.compile(r"[^;{]*\{").match(text, close + 1)
        if brace:
            out.setdefault(name, []).append((text[at + 1:close], text[brace.end() - 1:_closing(text, brace.end() - 1, "{}")]))
    return out


def _chained(text):
    names = set(re.findall(r"launch_chained\(\s*(\w+)", text)) - {"k"}
    for m in re.finditer(r"launch_chained\(\s*k\b", text):  # constexpr auto k = kernel<T>
        names.add(re.findall(r"constexpr auto k = (\w+)", text[:m.start()])[-1])
    return names


def test_chained_kernels_do_not_promise_read_only_data():
    text = _sources()
    funcs, todo = _functions(text), list(_chained(text))
    assert {"front_params_kernel", "flat_compress_kernel", "predict_compress_both_kernel", "leftover_fill_kernel",
            "shuffle_last_block_kernel", "bitshuffle_kernel", "encode_chunks_kernel", "scan_stream_kernel",
            "gather_stream_kernel"} <= set(todo)
    todo.append("write_trailer")  # called through a functor
    seen, bad = set(), []
    while todo:
        name = todo.pop()
        if name in seen or name not in funcs:
            continue
        seen.add(name)
        for params, body in funcs[name]:
            for p in re.findall(r"const\s+[\w:<>\s]+\*\s*__restrict__\s*(\w+)", params):
                if p not in FIELD:
                    bad.append((name, p))
            for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+)", body):
                if arg not in FIELD:
                    bad.append((name, "__ldg " + arg))
            todo += re.findall(r"\b(\w+)\s*(?:<[\w\s,()]*>)?\s*\(", body)
    assert {"shuffle_item", "chunk_is_zero", "scan_chunks", "gather_copy", "compress_tile"} <= seen
    assert not bad, bad


def test_field_is_complete_before_the_first_chained_kernel():
    text = _sources()
    assert not {"front_kernel", "params_kernel", "set_double_kernel"} & _chained(text)
    assert re.search(r"front_kernel<T><<<", text)
