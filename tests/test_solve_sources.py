"""What the solves' kernels must not do and no run shows reliably, checked on their source."""
import os

CSRC = os.path.join(os.path.dirname(__file__), "..", "gschism_b200", "csrc")


def test_phase_b_preload_does_not_read_the_flag_being_cleared():
    """k_jcg64: between phase A, where one thread clears Part::on, and the barrier behind it, no thread reads
    the flag."""
    text = open(os.path.join(CSRC, "jcg64.cu")).read()
    loop = text[text.index("for (int it = 0;; it++)"):]
    preload = loop[loop.index("// ---- B:"):loop.index("SYNC64();")]
    assert "first_on" in preload and ".on" not in preload
