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
    assert len(re.findall(r"bulk_load_row\([^;]*, nullptr\);", text)) == 1
    assert not re.search(r"try_wait|row_landed|await_row|clock64", text)
    assert not re.search(r"\breturn;", text[:text.index("cudaError_t rq_launch_wquant")])


def test_rotation_has_none_either():
    text = code("rq_act.cu")
    assert len(re.findall(r"^ {4}bulk_load_row\([^;]*, prm\.status\);", text, re.M)) == 1
    body = text[text.index("rq_act_kernel(const ActParams prm)"):]
    assert not re.search(r"\breturn;", body[:body.index("if (prm.a8 == nullptr) return;")])


def test_the_wait_without_a_status_word_ends_with_the_row():
    text = code("rq_act_dev.cuh")
    wait = text[text.index("void await_row("):text.index("void bulk_load_row(")]
    assert re.search(r"\} else if \(__syncthreads_or\(late\)\) \{.*cp\.async\.wait_all", wait, re.S) and "return" not in wait
