"""How many rows of logits the loss holds at a time."""
import pytest

from pisceslx_b200.ops.loss import rows_at_once


@pytest.mark.parametrize("T,V,H,rows", [
    (0, 1000, 64, 0), (1, 154856, 1024, 1), (2048, 154856, 4096, 2048),      # one chunk as before
    (2331, 154856, 1024, 2331), (8192, 32000, 4096, 8192),                   # no more than several chunks take, or than 2 GB
    (2730, 154856, 1024, 2730), (2731, 154856, 1024, 2048), (8192, 154856, 4096, 2048)])
def test_rows_at_once(T, V, H, rows):
    assert rows_at_once(T, V, H) == rows
