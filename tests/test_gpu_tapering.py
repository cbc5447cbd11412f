"""The FP64 segmented guide, which passes over the segments that certainly
hold a straight flight (FP32 bounds, csrc/components.cuh: taper_quiet),
against the CPU oracle's segment-by-segment loop on the same stream: every
slot of every neutron within 1e-12 relative (the denominator floored at the
slot's RMS), identical exit component -- the bound of the FP64 parity tests,
which the fewer steps between two reflections leave in place."""

import numpy as np
import pytest
import torch

from acc_gb300 import engine, instruments
from helpers import oracle_run, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    torch.cuda.init()
    yield


# segment counts around the block size of the quiet blocks (16) and the count
# that switches them on (256), and a guide without joints
@pytest.mark.parametrize("nseg", [1, 2, 17, 255, 256, 273])
@pytest.mark.parametrize("m", [6.0, -2.0, 0.0])
def test_fp64_segmented_guide_matches_the_oracle(nseg, m):
    n, seed = 4000, 31

    def build():
        return instruments.tapered_guide_chain(nseg=nseg, length=7.3, mx=m,
                                               my=6.0)

    out, last = engine.replay(engine.chain_for_instrument(build()), n,
                              seed=seed, floattype="float64")
    _, stats, ref, ref_last = oracle_run(build(), n, seed=seed, record=True)
    assert stats["processed"] == n
    np.testing.assert_array_equal(last.cpu().numpy(), ref_last)
    assert rel_err(out.cpu().numpy(), ref).max() <= 1e-12
