"""The layer kernel's RMSNorm scale over the sizes a residual can have: inv_sqrt_to_float's step up to mean squares of 2^100 and the expression itself
above (eps keeps the argument over 1e-6, so the lower end of the step's range is not reached). Bit for bit against the oracle. What its guard lets
through near the middle between two floats: test_norm_scale_host.py."""
import numpy as np
import pytest

import oracle_lib as ol
from warpdecode_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-5, 1.0, 3e7, 1.1e15, 1.2e15, 1e18])      # mean squares around 2^100 = 1.27e30 at 1.1e15 and 1.2e15
def test_stack_step_norm(oracle, scale):
    import warpdecode_b200 as wd
    m = synth.make_moe_block(3, 512, 256, 16, 4, 256)
    eng = wd.Engine(512, 256, 16, 4, 256, 1)
    eng.load_block(0, m)
    for seed in range(6):
        x = (np.random.Generator(np.random.PCG64(seed)).standard_normal(512) * scale).astype(np.float32)
        res = eng.stack_step_host(x)
        want = (x + oracle.moe_block(m, oracle.rmsnorm(x, None, 1e-6))["out"]).astype(np.float32)
        assert np.array_equal(ol.fbits(res), ol.fbits(want))
    assert eng.device_status() == 0
    eng.close()
