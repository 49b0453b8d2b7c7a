"""The hand-overs inside the resident solve (csrc/cgres.cuh), explored on the CPU:
every interleaving of the warps that meet there, with the number of buffers the
kernel declares.
"""

import re

from conftest import REPO

SRC = (REPO / "toptimization_b200" / "csrc" / "cgres.cuh").read_text()


def _buffers():
    """Copies of {alpha, beta, go on} in a CTA's shared memory."""
    m = re.search(r"__shared__ double s_ab(?:\[(\d+)\])?\[3\]", SRC)
    return int(m.group(1) or 1)


def test_coefficients_wait_for_every_warp_that_reads_them():
    """A CTA that does not collect the sums itself, with one group of nodes and
    one empty group. A warp of the first publishes its sums of exchange e, gets
    that exchange's coefficients (they come after its sums) and writes them for
    the CTA; both meet at a barrier and read them. The empty group publishes
    nothing, so nothing but the buffers keeps the next exchange's coefficients
    from a read that is late."""
    last, copies = 5, _buffers()
    # steps of the writer: 3 (e - 1) + (write, barrier, read); of the reader: 2 (e - 1) + (barrier, read)
    seen, todo = set(), [(0, 0, (0,) * copies)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        w, r, buf = state
        we, ws, re_, rs = w // 3 + 1, w % 3, r // 2 + 1, r % 2
        if we <= last and ws == 0:
            todo.append((w + 1, r, tuple(we if i == we % copies else b for i, b in enumerate(buf))))
        if we <= last and ws == 2:
            assert buf[we % copies] == we
            todo.append((w + 1, r, buf))
        if we <= last and ws == 1 and rs == 0 and re_ == we:  # both at the barrier
            todo.append((w + 1, r + 1, buf))
        if re_ <= last and rs == 1:
            assert buf[re_ % copies] == re_, "a warp reads the coefficients of a later exchange"
            todo.append((w, r + 1, buf))
    assert any(w == 3 * last and r == 2 * last for w, r, _ in seen)


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
