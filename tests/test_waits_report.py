"""CPU: no entry point gives up silently.  A bounded wait of a kernel ends, when it runs out, in a status word that the caller reads;
the entry points without such a word (weight conversion, the rotation alone) run code that waits for nothing.  Read from the
sources, since the wait itself cannot be made to run out by a caller."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc")


def code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_weight_conversion_waits_for_nothing():
    assert not re.search(r"mbarrier|bulk_load_row|try_wait|clock64", code("rq_wquant.cu"))


def test_rotation_without_a_status_word_waits_for_nothing():
    text = code("rq_act.cu")
    calls = [m.start() for m in re.finditer(r"bulk_load_row\(", text)]
    assert len(calls) == 1
    assert "if (prm.status != nullptr) {" in text[calls[0] - 120:calls[0]]
