"""The mailbox of the register-resident Jacobi sweep under the memory model of PTX,
where a vector access is one access per element in any order: an entry whose
stamps a reader finds renewed holds the numbers that were sent with them,
whatever the interleaving of its elements' stores and loads.  The element width
is the one that the kernel's source names."""
import itertools
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qaintensor.jl_gb300", "csrc",
                   "k_jacobi.cu")


def access(op):
    """(ordering, elements, words per element) of the mailbox's store or load."""
    text = open(SRC).read()
    body = text[text.index("mail_" + {"st": "store", "ld": "load"}[op] + "("):]
    m = re.search(r'"%s\.([\w.]+)\.global\.v(\d)\.[bu](\d+) ' % op, body)
    return m.group(1), int(m.group(2)), int(m.group(3)) // 32


def test_a_renewed_stamp_comes_with_its_number():
    (st_order, st_n, st_words), (ld_order, ld_n, ld_words) = access("st"), access("ld")
    # strong accesses (volatile counts as relaxed at system scope)
    assert {st_order, ld_order} <= {"relaxed.gpu", "relaxed.sys", "volatile"}
    assert st_n * st_words == ld_n * ld_words == 4  # number, stamp, number, stamp
    old, new = ["re0", 1, "im0", 1], ["re1", 2, "im1", 2]

    def pieces(n, words):
        return [range(words * i, words * (i + 1)) for i in range(n)]

    seen = 0
    events = [("st", p) for p in pieces(st_n, st_words)] + [("ld", p) for p in pieces(ld_n, ld_words)]
    for order in itertools.permutations(events):
        memory, got = list(old), [None] * 4
        for kind, piece in order:
            for w in piece:
                if kind == "st":
                    memory[w] = new[w]
                else:
                    got[w] = memory[w]
        if got[1] == got[3] == 2:
            seen += 1
            assert got == new, order
    assert seen
