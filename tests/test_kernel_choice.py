"""Which kernel a call takes, where the wrappers choose by sizes: checked on the CPU at sizes that were measured."""
import pytest

from garlic_inference_b200.ops import kernels


@pytest.mark.parametrize("lens, heads, d, channel, chunks", [
    ([2048], 16, 128, True, True), ([100] * 2, 16, 128, True, True), ([800] * 5, 16, 128, True, True), ([500] * 8, 16, 128, True, True),
    ([600] * 3, 16, 128, False, True), ([300] * 4, 8, 64, False, True),
    # many blocks hide the chain of token by token: 545 us, 698 in chunks; 295 and 313; 652 and 742; 77 and 95
    ([500] * 16, 16, 128, False, False), ([600] * 6, 16, 128, False, False), ([500] * 16, 16, 128, True, False), ([300] * 16, 8, 64, False, False),
    ([100] * 8, 16, 128, True, False), ([40], 16, 128, True, False)])
def test_delta_rule_in_chunks_or_token_by_token(lens, heads, d, channel, chunks):
    assert kernels._delta_in_chunks(sum(lens), len(lens), heads, d, d, channel) == chunks


@pytest.mark.parametrize("n, heads, cut", [(1, 8, False), (2, 8, False), (4, 16, False), (8, 4, False), (8, 8, True), (16, 4, True), (32, 8, True),
                                           (64, 4, True), (33, 8, False), (65, 2, False), (64, 8, False)])
def test_decode_attention_in_slices_of_one_length(n, heads, cut):
    places = kernels.decode_places_tcgen05(n, heads)
    assert (places > 0) == cut and (not cut or n <= places <= 16 * n)
