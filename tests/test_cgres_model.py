"""The hand-overs inside the resident solve (csrc/cgres.cuh), explored on the CPU:
every interleaving of the warps that meet there, with the number of buffers the
kernel declares.
"""

import re

from conftest import REPO

SRC = (REPO / "toptimization_b200" / "csrc" / "cgres.cuh").read_text()


def test_coefficients_wait_for_every_warp_that_reads_them():
    """A CTA that does not collect the sums itself, with one group of nodes and
    one empty group. A warp of the first publishes its sums of exchange e, gets
    that exchange's coefficients (they come after its sums) and writes them for
    the CTA; both meet at a barrier and read them. The empty group publishes
    nothing, so a late read of it has to be kept from the next exchange's
    coefficients otherwise: by a barrier after the reads, or by a second buffer."""
    m = re.search(r"__shared__ double s_ab(?:\[(\d+)\])?\[3\]", SRC)
    copies = int(m.group(1) or 1)
    reads = SRC.index("alpha = s_ab[0];") if copies == 1 else 0
    held = re.search(r"if \(!lead && unfilled\) __syncthreads\(\);", SRC[reads:]) is not None
    last = 5
    after = ["barrier"] if held else []
    writer = [(op, e) for e in range(1, last + 1) for op in ["write", "barrier", "read"] + after]
    reader = [(op, e) for e in range(1, last + 1) for op in ["barrier", "read"] + after]
    seen, todo = set(), [(0, 0, (0,) * copies)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        w, r, buf = state
        wop, we = writer[w] if w < len(writer) else (None, 0)
        rop, re_ = reader[r] if r < len(reader) else (None, 0)
        if wop == "write":
            todo.append((w + 1, r, tuple(we if i == we % copies else b for i, b in enumerate(buf))))
        elif wop == "read":
            assert buf[we % copies] == we
            todo.append((w + 1, r, buf))
        elif wop == "barrier" and rop == "barrier":
            assert we == re_
            todo.append((w + 1, r + 1, buf))
        if rop == "read":
            assert buf[re_ % copies] == re_, "a warp reads the coefficients of a later exchange"
            todo.append((w, r + 1, buf))
    assert any(w == len(writer) and r == len(reader) for w, r, _ in seen)


def _element_bytes(fn):
    """Bytes of one element of the vector access in `fn`: what the memory model
    moves in one piece."""
    m = re.search(rf"{fn}\(.*?\.global\.v(\d)\.[bu](\d+)", SRC, re.S)
    assert int(m.group(1)) * int(m.group(2)) == 128
    return int(m.group(2)) // 8


def test_exchanged_word_is_taken_only_when_all_of_it_is_there():
    """A double travels as 16 bytes, {low word, epoch, high word, epoch}, whose
    elements may become visible one by one; the reader takes it when both
    epochs are the current ones. Whatever mix of an old and a new word it
    sees, what it takes has to be the new value."""
    size = min(_element_bytes("ll_store"), _element_bytes("ll_load"))
    old, new = ("old low", 1, "old high", 1), ("new low", 3, "new high", 3)
    n = 16 // size
    for arrived in range(1 << n):
        word = tuple((new if arrived >> (4 * k // size) & 1 else old)[k] for k in range(4))
        if word[1] == word[3] == 3:
            assert (word[0], word[2]) == ("new low", "new high"), "an epoch came before its data"
