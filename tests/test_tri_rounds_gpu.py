"""The triangular solve around a round of the block's seven warps (224
positions) and two, on chains that take a chunk's every position, bit for bit
against the CPU restatement."""
import pytest

from test_tri_chunks_gpu import test_trsv_chunks_and_division as chunks_and_division

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", ["f64", "c64"])
@pytest.mark.parametrize("n,reach", [(223, 1), (224, 1), (225, 1), (447, 2), (448, 1), (449, 1), (7168, 33), (7169, 31)])
def test_rounds_of_seven_warps(gpu, n, reach, t):
    chunks_and_division(gpu, n, reach, t)
