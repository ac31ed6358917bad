"""Which way a step's recurrences go (host rules; no GPU)."""
import pytest

from photon_infer_b200.kernels import ops


@pytest.mark.parametrize("lens,heads", [([777], 16), ([2048], 16), ([640], 32), ([700, 700], 16), ([70] * 24, 16)])
def test_forget_and_write_takes_no_chunks(lens, heads):
    """Its outputs were further from 64 bits there, and write gates near 1 made a step several times longer."""
    assert not ops.linrec_chunks_supported("forget_write", 128, 128, lens, heads)
