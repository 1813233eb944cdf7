"""Two rules of the peel's memory accesses that no run can show, read from the
sources: one width of atomics on a packed word, and no plain access to a word
that another thread may be writing in the same step."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "pargridcpu_b200", "csrc")


def body(source, name):
    """The body of the function `name`, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, source)).read())
    at = re.search(r"\b%s\([^;{]*\)\s*\{" % name, text)
    depth, end = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at.end():end]


def test_late_form_decrements_whole_words():
    """An item of one column and an item of several meet on the same degree
    and count words: both must use 64-bit atomics."""
    text = body("late.cu", "lt_item_run")
    atomics = re.findall(r"atomic\w+\(\s*([^;]*)", text)
    packed = [a for a in atomics if "j.deg" in a or "j.cnt" in a]
    assert packed
    for a in packed:
        assert "uint32_t*" not in a, a


def test_masks_are_not_read_plainly_while_owners_clear_them():
    """An expansion tests neighbours' masks while other threads clear columns
    in theirs."""
    for source, name in (("peel.cu", "visit"), ("peel.cu", "retire"), ("late.cu", "lt_filter"),
                         ("late.cu", "lt_item_run")):
        assert "j.M[" not in body(source, name), (source, name)


def test_hand_over_reads_only_written_degrees():
    """The first scan writes no degree word whose columns all leave the node
    there, and the scratch is not cleared: the hand-over to the late form
    copies a word only if one of its columns is left."""
    text = body("late.cu", "k_lt_degrees")
    assert re.search(r"if \(\(M >> \(4 \* q\)\) & 15u\) d = src\[", text)
