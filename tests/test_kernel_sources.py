"""Orders inside the kernels that a run on the GPU cannot show, because they hold by luck when they are missing: read from the
sources (no GPU needed)."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tesseract_b200", "csrc")


def code_of(name):
    with open(os.path.join(CSRC, name)) as handle:
        return re.sub(r"//[^\n]*", "", handle.read())


def test_tensor_memory_that_a_product_used_is_touched_behind_a_fence():
    """attention_tcgen05: a softmax thread that waited for a product's commit (``o_full``) reads or writes what the product
    used (its probabilities, its output) only behind ``tcgen05.fence::after_thread_sync``."""
    code = code_of("attention_tcgen05.cu")
    softmax = code[code.index("const uint32_t lane_base"):]
    events = re.finditer(r"(?P<wait>mbar_wait\(o_full)|(?P<fence>tc_fence_after\(\))|"
                         r"(?P<touch>tmem_(?:load|store)\w*\(tmem_[op]\b)", softmax)
    waiting, waits, touches = False, 0, 0
    for event in events:
        if event["wait"]:
            waiting, waits = True, waits + 1
        elif event["fence"]:
            waiting = False
        else:
            touches += 1
            line = softmax[:event.start()].count("\n") + code[:code.index("const uint32_t lane_base")].count("\n") + 1
            assert not waiting, f"line {line}: no fence between the wait for a product and this access"
    assert waits >= 4 and touches >= 8
