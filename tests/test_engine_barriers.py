"""The group exchange of the N4 engine, read from its source (csrc/n4_engine.cuh).

Pass A leaves each CTA's sums in that CTA's one statistics slot, the others read
them after a group barrier.  The slot may be written again only after a further
group barrier: between two passes A there has to be one, in every order the
statements of `Engine::run` can be taken.  `fit_step` and `contract` hold one
each, `g.sync()` is one.
"""
import os
import re

from conftest import ROOT


def body(src, head):
    """The brace-balanced block that follows `head`."""
    i = src.index("{", src.index(head))
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        j += 1
        if depth == 0:
            return src[i:j]


def source():
    with open(os.path.join(ROOT, "cuda-n4_b200", "csrc", "n4_engine.cuh")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


STEP = re.compile(r"(?:!|\b)(pass_a|fit_step|contract<false>|g\.sync)\s*\(")


def steps(text):
    return [m.group(1) for m in STEP.finditer(text)]


def written_again_at_once(order):
    return [k for k in range(1, len(order)) if order[k] == order[k - 1] == "pass_a"]


def test_a_barrier_lies_between_two_passes_a():
    src = source()
    assert "g.sync()" in body(src, "bool contract(Fin &&fin)")
    assert "contract<true>" in body(src, "bool fit_step(")
    run = body(src, "void run(const VolJob &job)")
    levels = body(run, "for (int level = 0;")
    trial = steps(body(levels, "for (int arm = 0;"))
    main = steps(body(levels, "for (;;)"))
    start = steps(levels[:levels.index("for (int arm = 0;")])
    assert start.count("contract<false>") == 1 and trial.count("pass_a") == 2 and main == ["pass_a", "fit_step"]
    for k in (0, 1, 3):   # main iterations, the pass A that ends them, the next level
        for arms in (0, 2):
            order = start + trial * arms + main * k + ["pass_a"] + start + main
            assert not written_again_at_once(order), order
