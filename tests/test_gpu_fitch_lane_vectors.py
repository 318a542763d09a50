"""Fitch distances at the lengths where a lane's share grows to two, three and four
vectors, each a kernel of its own (csrc/fitch_sankoff.cu), against a count on the CPU."""
import pytest

from tests.test_gpu_fitch_rows import test_distances_at_vector_and_batch_edges as distances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [400, 1023, 1024, 1025, 1536, 1537, 2000])
def test_one_to_four_vectors_a_lane(length):
    distances(length)
