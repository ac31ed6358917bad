"""Which way a step's recurrences go (host rules; no GPU)."""
import pytest

from photon_infer_b200.kernels import ops


@pytest.mark.parametrize("lens,heads", [([777], 16), ([2048], 16), ([640], 32), ([700, 700], 16), ([70] * 24, 16)])
def test_forget_and_write_takes_no_chunks(lens, heads):
    """Its outputs were further from 64 bits there, and write gates near 1 made a step several times longer."""
    assert not ops.linrec_chunks_supported("forget_write", 128, 128, lens, heads)


@pytest.mark.parametrize("mode,heads,dim,blocks,lens,chunks", [
    # few chunks that hold little, and one block more than a round: the segments (us, segments and chunks: 61 and 76, 60 and 76, 45 and 62)
    ("decay_rows", 32, 128, 2, [130] * 3, False), ("decay_rows", 16, 128, 2, [130] * 5, False), ("state_space", 32, 128, 2, [130] * 3, False),
    # requests that fill the GPU uncut, in one pass (282 and 460, 123 and 166, 126 and 182)
    ("decay_rows", 64, 64, 1, [700] * 4, False), ("decay_rows", 64, 64, 1, [300] * 3, False), ("state_space", 80, 128, 1, [300] * 3, False),
    # few rows a head (116 and 153, 100 and 128)
    ("decay_rows", 32, 32, 1, [2048], False), ("state_space", 32, 32, 1, [2048], False),
    # a round that is full, and several (112 and 44, 115 and 78, 176 and 102, 118 and 74, 183 and 94, 155 and 82)
    ("decay_rows", 16, 128, 2, [1152], True), ("decay_rows", 16, 128, 2, [1200], True), ("decay_rows", 16, 128, 2, [2048], True),
    ("decay_rows", 32, 128, 2, [640], True), ("matrix_memory", 16, 128, 2, [2048], True), ("state_space", 16, 128, 2, [2048], True),
    ("decay_rows", 16, 128, 2, [640], True), ("matrix_memory", 16, 128, 2, [1284, 1531], True), ("decay_rows", 32, 128, 2, [700, 700], True)])
def test_chunks_where_their_rounds_are_less_than_the_passes(mode, heads, dim, blocks, lens, chunks):
    """The B200's 148 multiprocessors; `blocks`: of a segment and head."""
    assert ops.linrec_chunks_faster(mode, dim, tuple(lens), heads, blocks, 148) == chunks


def test_an_unknown_mode_is_an_argument_error():
    import torch
    from photon_infer_b200.errors import PhotonError
    rows = torch.zeros(1024, 16 * 128)
    with pytest.raises(PhotonError):
        ops.linrec_segments("no such mode", rows, rows, rows, None, None, None, None, None, None, 0.0, 1.0, torch.zeros(2, dtype=torch.int32),
                            torch.zeros(1, dtype=torch.int32), torch.zeros(1, 16 * 128 * 128), rows, [1024], 16, 16, 128, 128, None)
