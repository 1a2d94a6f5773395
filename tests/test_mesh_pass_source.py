"""The spread mesh is zero between passes.  A spread and the convolution that clears it go through one function,
which marks the mesh before the spread and unmarks it once the convolution is queued: an error in between (a
plan, a matrix or a transform that fails) then leaves a mark, not a spread that the next energy adds to its own.
Such errors cannot be brought about on a working GPU, so this reads the source."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "dmff_b200", "csrc", "engine.cu")


def _code():
    return re.sub(r"//[^\n]*", "", open(SRC).read())


def _body(code, head):
    i = code.index("{", code.index(head))
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(code[j], 0)
        j += 1
        if depth == 0:
            return code[i:j]


def test_mesh_pass_marks_before_and_unmarks_after():
    body = _body(_code(), "int mesh_pass(")
    order = [body.index(x) for x in ("clean_mesh<T>", "grid2_dirty = true", "spread();", "mesh_convolve<T>", "return st;\n    h->grid2_dirty = false")]
    assert order == sorted(order)


def test_every_spread_and_convolution_goes_through_it():
    code = _code()
    assert len(re.findall(r"mesh_convolve<T>\(", code)) == 1
    launches = [m.start() for m in re.finditer(r"k_spread\w*<T[^>]*><<<", code)]
    assert len(launches) == 4
    lambdas = [(m.start(), m.start() + len(_body(code[m.start():], "[&]"))) for m in re.finditer(r"auto spread = \[&\] \{", code)]
    assert len(lambdas) == len(re.findall(r"mesh_pass<T>\(h, s, .*, spread\)", code)) == 3
    for at in launches:
        assert any(a < at < b + 40 for a, b in lambdas), code[at:at + 80]
    # the persistent solve spreads by itself: marked before its launch
    assert re.search(r"grid2_dirty = true;\s*return cg_persistent\(", code)
