"""CPU: where the wait for a kernel's weights runs out, the block waits for them
once more before it gives its shared memory back (the copies may still be on
their way).  Read from the source: nothing is made to run out on a GPU."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_weights_are_waited_for_again():
    src = open(os.path.join(ROOT, "alamo_gb300", "csrc", "kernels_conv_march.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    assert re.search(r"ok = __all_sync\(0xffffffffu, mbar_wait\(wbar, 0\)\);\s*if \(!ok\) mbar_wait\(wbar, 0\);", src)
