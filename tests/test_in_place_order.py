"""The in-place unique: a block writes over places that lower blocks read, so
what it waits for (the lower blocks' posted totals) has to depend on everything
they read, in a way that the compiler cannot remove."""
import os
import re

SCAN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "glsl-tree-construction_gb300", "csrc",
                    "scan.cu")


def function(name):
    """The text of a function, without comments: from its name to the brace that closes it."""
    text = re.sub(r"//[^\n]*", "", open(SCAN).read())
    at = re.search(r"\b%s\s*\((?=[^;]*?\{)" % name, text).start()
    depth = 0
    for i in range(text.index("{", at), len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]


def test_total_depends_on_the_values():
    """The count takes in the values under a mask that only the launch knows to be 0."""
    body = function("row_unique_kernel")
    assert re.search(r"\buint32_t zero\)", body)  # a kernel argument
    used = re.search(r"cnt \+= [^;]*\bx & zero\);", body).start()
    assert body.index("x |= v[j]") < used < body.index("s_seg[warp] = cnt") < body.index("cs_block_prefix(")


def test_the_launch_passes_zero():
    assert re.search(r"launch_kernel\(L, kern, [^;]*L\.status, 0u\);", function("launch_row_unique"))
