"""Which prompt products run on tensor cores (wd_prompt_tile): the choice holds for products that were measured both ways, and what the rule leaves out."""
import pytest

import test_gpu_prompt_tc_tiles as tc
import warpdecode_b200 as wd

Q4, Q8 = wd.TYPE_Q4_0, wd.TYPE_Q8_0

# rows, cols, type, tokens; us of the product on mma.sync, and on tensor cores with tiles of 32, 48 and 64 tokens, its laying out included
MEASURED = [
    (4096, 2048, Q8, 97, 19.6, 24.4, 24.2, 25.6), (6144, 2048, Q8, 65, 19.8, 24.7, 27.2, 29.3), (2048, 2048, Q8, 256, 20.3, 24.1, 22.1, 23.4),
    (4096, 2048, Q4, 97, 18.1, 21.2, 22.6, 24.5), (2048, 2048, Q4, 65, 12.2, 18.7, 20.7, 22.7), (2048, 5632, Q4, 256, 45.0, 48.1, 51.8, 55.8),
    (2048, 5632, Q4, 80, 29.6, 47.4, 51.7, 55.9), (11264, 2048, Q8, 33, 29.3, 36.2, 29.1, 31.2),
]


@pytest.mark.parametrize("rows,cols,wtype,tokens,other,t32,t48,t64", MEASURED)
def test_no_product_is_given_to_the_slower_kernel(rows, cols, wtype, tokens, other, t32, t48, t64):
    took = {0: other, 32: t32, 48: t48, 64: t64}[wd.prompt_tile(rows, cols, wtype, tokens)]
    assert took <= 1.02 * other and took <= 1.05 * min(other, t32, t48, t64)


def test_what_pays_and_what_is_left_out():
    assert wd.prompt_tile(16384, 2048, Q4, 480) == 64       # 247 us on mma.sync, 150 on tensor cores
    for wtype in (Q4, Q8):
        for rows in (64, 1024, 28672):
            assert wd.prompt_tile(rows, 992, wtype, 512) == 0 and wd.prompt_tile(rows, 2048, wtype, 32) == 0
    with pytest.raises(wd.WdError):
        wd.prompt_tile(1024, 1000, Q4, 64)


@pytest.mark.parametrize("case", tc.CASES)
def test_the_gpu_cases_run_where_they_say(case):
    assert tc.tiles_of(wd, *case[:7]) == case[7]
