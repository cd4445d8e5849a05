"""Orders and bounds in the kernels that no run can show to be missing without risking a hang:
read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neuzip_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_tensor_memory_is_taken_between_the_wait_and_the_trigger():
    # launched while the kernel before it still runs: a CTA that holds tensor memory while it
    # waits, or lets its successor in before it has its own, can wait for ever
    text = source("nz_linear.cu")
    body = text[text.index("linear_kernel(const LinearArgs p"):text.index("linear_finish_kernel(")]
    wait, alloc = body.index("griddepcontrol.wait"), body.index("tcgen05.alloc")
    barrier = body.index("__syncthreads()", alloc)
    assert body.count("griddepcontrol.wait") == body.count("tcgen05.alloc") == 1
    assert wait < alloc < barrier < body.index("griddepcontrol.launch_dependents")


def test_waits_give_a_slow_copy_a_million_tries():
    text = source("nz_decode_core.cuh")
    tries = re.search(r"kMaxWaitIters = 1u << (\d+);", text)
    hint = re.search(r"kWaitHintNs = (\d+);", text)
    assert int(tries.group(1)) >= 20                               # how early a try returns is open
    assert int(hint.group(1)) << int(tries.group(1)) <= 2 << 30    # and the wait stays bounded
