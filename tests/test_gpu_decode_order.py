"""Decode attention that takes its requests longest first: more pairs of request and key/value head than the kernel has
blocks (two per multiprocessor), up to 128 requests."""
import pytest

from test_gpu_kernels import _decode_attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("requests,n_q,n_kv,chunk", [
    (38, 24, 8, 2), (75, 8, 4, 64), (127, 4, 4, 1), (128, 6, 3, 3), (129, 6, 3, 3)])
def test_requests_of_mixed_lengths(requests, n_q, n_kv, chunk):
    """Lengths that rise, fall and repeat, so that the order of work is neither the step's nor its reverse; each request
    must still find its own queries, pages and partial results."""
    lens = [1 + (i * 197) % 611 if i % 3 else 64 * (1 + i % 5) for i in range(requests)]
    _decode_attention_case(n_q, n_kv, 64, 16, None, lens, [1] * requests, chunk)


def test_requests_with_a_window():
    lens = [2000 - 40 * i if i % 2 else 30 + 7 * i for i in range(48)]
    _decode_attention_case(16, 8, 128, 16, 150, lens, [1] * 48, 2)
