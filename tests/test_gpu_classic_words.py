"""GPU: misaligned classic jobs on enough columns for the word kernel
(classic_rules.hpp), with the checks of test_gpu_classic_unaligned.py: lengths
from the shortest it takes to several tiles, every remainder of a word and of a
tile's last row of threads, one to twenty outputs; and the launch that is just too
small for it."""
import pytest

import test_gpu_classic_unaligned as unaligned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,m,length", [(1, 1, 1645), (3, 2, 1649), (4, 4, 2051), (5, 3, 3079), (10, 4, 4103),
                                        (12, 4, 4107), (16, 4, 8203), (21, 4, 8211), (10, 4, 100003)])
@pytest.mark.parametrize("shift", [0, 5])
def test_up_to_four_outputs(k, m, length, shift):
    unaligned.test_packed_odd_shards(k, m, length, shift, 704 << 10)


@pytest.mark.parametrize("k,m,length", [(7, 8, 2573), (9, 5, 4101), (30, 9, 12305), (50, 20, 100003)])
def test_more_outputs(k, m, length):
    unaligned.test_packed_odd_shards(k, m, length, 3, 1 << 20)


@pytest.mark.parametrize("k,m,length,stripes", [(10, 4, 4103, 175), (6, 3, 720897 - 2, 1), (9, 5, 4101, 255)])
def test_one_stripe_less(k, m, length, stripes):
    unaligned.test_packed_odd_shards(k, m, length, 1, (stripes - 1) * length)


@pytest.mark.parametrize("k,m", [(4, 2), (10, 4), (7, 8)])
def test_one_long_stripe(k, m):
    """The accumulating and the storing calls by words."""
    unaligned.test_packed_odd_shards(k, m, 1100003, 2, 0)
