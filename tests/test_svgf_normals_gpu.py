"""Normals whose length overflows single precision: finite, so their pixels are
valid, but they normalise to zero and weigh nothing with any other."""
import numpy as np
import pytest

import svgf_cases as S
from renderingengine_b200.svgf import SvgfReconstruction
from test_svgf_gpu import _cfg_pair, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e18, 3e19, 1e30])
def test_huge_normals_match_oracle(native, oracle, scale):
    native_cfg, py_cfg = _cfg_pair(atrous_iterations=5)
    w, h = 48, 33
    gpu = SvgfReconstruction(w, h, 2, py_cfg)
    ora = oracle.OracleSvgf(w, h, 2, native_cfg)
    for gb, sig, fi, trig in S.sequence(w, h, 4, 21, hostile=False):
        gb = gb.copy()
        with np.errstate(over="ignore"):  # twice 1e30 is not finite: those pixels are not valid
            gb["world_normal"][5:20, 8:30] *= np.float32(scale)
            gb["world_normal"][::4, ::5] *= np.float32(scale)
        _compare(gpu.process(gb, sig, fi, trig), ora.process(gb, sig, fi, trig), f"frame {fi}")
