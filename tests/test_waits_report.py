"""CPU: no entry point gives up silently.  A bounded wait of a kernel ends, when it runs out, in a status word that the caller reads;
the entry points without such a word (weight conversion, the rotation alone) load their rows in the way that needs none: it
copies the row again instead of giving up.  Read from the sources, since a caller cannot make the wait run out."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc")


def code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_weight_conversion_has_no_way_out():
    text = code("rq_wquant.cu")
    assert text.count("load_row_surely(") == 1 and not re.search(r"bulk_load_row|try_wait|row_landed|clock64", text)
    kernels = text[:text.index("cudaError_t rq_launch_wquant")]
    assert not re.search(r"\breturn;", kernels)


def test_rotation_without_a_status_word_has_none_either():
    text = code("rq_act.cu")
    at = text.index("bulk_load_row(")
    assert text.count("bulk_load_row(") == 1 and "if (prm.status != nullptr) {" in text[at - 60:at]
    assert re.match(r"bulk_load_row\([^;]*;\s*\} else \{\s*load_row_surely\(", text[at:])
