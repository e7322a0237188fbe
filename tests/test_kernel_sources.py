"""CPU checks of rules that the kernels' sources have to keep and that no run can show."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spargeattn_b200", "csrc")


def _waiting_kernels():
    """(name, parameters, body) of every kernel that may run beside the one before it."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__.*?(\w+_kernel)\((.*?)\)\s*\{\n(.*?)\n\}\n", text, flags=re.S):
            if "pdl_wait" in m.group(3):
                found.append(m.groups())
    return found


def test_kernels_that_wait_for_the_one_before_do_not_claim_constant_inputs():
    kernels = _waiting_kernels()
    assert {k[0] for k in kernels} >= {"prep_combine_kernel", "prep_second_kernel", "select_kernel", "mask_to_lut_kernel", "attn_kernel"}
    for name, parameters, _ in kernels:
        for parameter in parameters.split(","):
            assert not ("const" in parameter and "__restrict__" in parameter), (name, parameter)
