"""The FP32 expansion of one species with many neighbours (about 51), on both
sides of the rule that picks its kernel by the sums a lane would keep: 8 and 16
(chunks), 24 and 48 (registers), 64 and 96 (chunks again); 16 copies of a box
(1 920 centres, more than get a block each).

Tolerance: the FP32 features' bar, 1e-5 of the largest value."""
import pytest

from test_gpu_expansion_channels import copies_match_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l", [(5, 4), (8, 6), (12, 6), (16, 8), (14, 10), (16, 12)])
def test_one_species(n, l):
    copies_match_oracle(n, l, (8,), 8.5)
