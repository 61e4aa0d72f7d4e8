"""CPU: a ragged plan is destroyed in an order that no launch in flight can miss."""
import os

from conftest import ROOT


def test_host_word_outlives_the_launches():
    """The last CTA of a launch that gave up writes the plan's pinned word; freeing device
    memory waits for the launch, freeing pinned memory is not promised to."""
    text = open(os.path.join(ROOT, "wgls-rs-fft_gb300", "csrc", "fft_ragged.cu")).read()
    body = text[text.index("void ragged_plan_free("):]
    body = body[:body.index("\n}")]
    assert "cudaFreeHost" in body
    assert -1 < body.find("meta.release()") < body.index("cudaFreeHost")
