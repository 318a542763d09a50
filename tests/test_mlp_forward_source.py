"""csrc/mlp_forward.cu, as text.  The lanes of a warp part in waits, in what one
thread does alone and in loads and stores of rows past the last; a __syncwarp()
brings them together before the next .aligned instruction (a tensor-memory load,
store or wait, the release of tensor memory, and the main warps' bar.red), and no
lane leaves a loop of such instructions by what it alone has read."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "poyd_gb300", "csrc", "mlp_forward.cu")
PART = r"\bwait\(bar|\bget_x\(|\bput_x\(|if \((tid|lane) == 0\)|if \(h\)|if \(\*dead\)"
TOGETHER = r"__syncwarp\(\);"
ALIGNED = r"m_epilogue<|m_head<|m_main_sync\(|m_ld32\(|m_st16\(|\.sync\.aligned"


def source():
    return re.sub(r"//[^\n]*", "", open(SRC).read())


def body(text, head):
    """The braces that follow `head`."""
    i = text.index("{", text.index(head))
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return text[i:j]


def test_lanes_come_together_before_aligned_instructions():
    text = source()
    for head in ("void m_epilogue(", "float m_head(", "k_mlp_forward("):
        code = body(text, head)
        if head == "k_mlp_forward(":  # from the loops on; before them, __syncthreads()
            code = code[code.index("quarter < 4) {"):]
        apart, seen = None, 0
        for m in re.finditer("(%s)|(%s)|(%s)" % (PART, TOGETHER, ALIGNED), code):
            word = m.group(0)
            if re.match(TOGETHER, word):
                apart = None
            elif re.match(PART, word):
                apart = word
            else:
                seen += 1
                assert apart is None, (head, apart, code[m.start():m.start() + 60])
        assert seen >= 1, head


def test_loops_end_for_the_whole_warp():
    assert not re.search(r"(for|while) \([^{]*!\*dead", source())
