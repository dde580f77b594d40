"""Where a kernel lets the next launch begin: host logic alone, by the source."""
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neurogrid_b200", "csrc")


def test_norm_and_convolution_lets_the_next_launch_begin_after_its_wait():
    """The step was slower with the launch than with the two it replaces where it let the next begin at its top."""
    text = open(os.path.join(CSRC, "input_conv.cu")).read()
    body = text[text.index("norm_conv_token_kernel(float*"):]
    assert body.index("ng_pdl_wait()") < body.index("ng_pdl_trigger()")
