"""Rules of the device code that no run can show to be broken, read from the sources (no GPU)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "q3_b200" / "csrc"


def test_values_exchanged_between_blocks_are_whole_64_bit_elements():
    """The tridiagonalisation's readers take a value as current when the step beside each half is.
    The PTX memory model keeps an element of a vector access whole, not the vector, so half and
    step have to share one 64-bit element."""
    text = (CSRC / "dense.cu").read_text()
    vectors = re.findall(r"\b(?:ld|st)\.volatile\.global\.(v\d\.\w+)", text)
    assert vectors and set(vectors) == {"v2.b64"}, vectors
