"""The exact merge on both sides of the line between word and byte reads (an image of 0.7 of the panorama's
2405 pixels): the same panoramas from images at a 4-byte boundary and off it."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("image", [(36, 46), (36, 47), (421, 4), (420, 4), (2, 842)])
@pytest.mark.parametrize("refs", [1, 4])
def test_both_sides_of_the_line(ss, native, image, refs):
    from test_gpu_merge_words import test_word_and_byte_reads_agree as reads_agree

    reads_agree(ss, native, 40, 32, image, refs)
