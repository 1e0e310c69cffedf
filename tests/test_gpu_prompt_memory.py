"""What a dense decoder takes of the GPU's memory for prompts on tensor cores: nothing where its prompts are too short or its rows too narrow for them,
a copy of the matrices that they read otherwise."""
import pytest

pytestmark = pytest.mark.gpu


def taken(hidden, heads, ffn, max_ctx):
    """Bytes that a decoder takes beside its matrices (held twice, in the file's form and for the step)."""
    import torch
    import warpdecode_b200 as wd
    torch.cuda.init()
    free = lambda: torch.cuda.mem_get_info()[0]
    wd.DenseDecoder(hidden, heads, heads // 4, 64, ffn, 96, 1, max_ctx).close()         # the context's own memory
    before = free()
    dec = wd.DenseDecoder(hidden, heads, heads // 4, 64, ffn, 96, 1, max_ctx)
    used = before - free()
    dec.close()
    weights = hidden * heads * 64 * 5 // 2 + 3 * hidden * ffn
    return used - weights * 18 // 32 * 2, weights


def test_short_prompts_hold_no_copy_of_a_layer():
    few, weights = taken(2048, 32, 8192, 32)
    many, _ = taken(2048, 32, 8192, 512)
    copy = weights * 5 // 8
    assert few < 24 << 20                       # 4 MB of workspace, caches, rounding of a dozen allocations to 2 MB
    assert copy < many < copy + (512 * 140 << 10) + (24 << 20)


def test_narrow_rows_hold_no_copy_of_a_layer():
    used, weights = taken(512, 8, 992, 512)     # every row has fewer than 1024 columns
    assert used < (512 * 40 << 10) + (24 << 20)
