"""The FP32-mixed 3-D form without z-boundary physics rounds no worse than the one with it.

Problems without z-boundary and corrected physics have operations of their own
(march_block32, stage3d_plain32); the others run stage3d_body32.  A fixed
temperature gradient of zero at reflecting z boundaries is what those
boundaries do anyway, but takes a problem to the other body: the same flow in
both, each held to FP64.  In a stratified layer at near rest one more rounding
of a flux shows in w as 1.4 times the error, so both make the same number of
them when the ratio, 1 but for the average over seeds, stays under 1.18,
half-way in powers.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from test_gpu_march_error import SEEDS, layer3d, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("visc", [True, False])
def test_no_larger_error(visc, monkeypatch):
    logs = []
    for seed in range(SEEDS):
        pr = layer3d(200 + seed)
        pr.params.viscosity_active = int(visc)
        want, _ = run(pr, fv._abi.FV_PREC_FP64, None, monkeypatch)
        got, _ = run(pr, fv._abi.FV_PREC_FP32_MIXED, None, monkeypatch)
        for side in ("zmin", "zmax"):
            setattr(pr.params, "bctc_" + side, fv._abi.FV_BCTC_FIXED_GRADIENT)
            setattr(pr.params, "bctc_%s_value" % side, 0.0)
        np.testing.assert_array_equal(run(pr, fv._abi.FV_PREC_FP64, None, monkeypatch)[0][3], want[3])
        ref, tx = run(pr, fv._abi.FV_PREC_FP32_MIXED, None, monkeypatch)
        assert tx == 16
        err = [np.linalg.norm(x[3] - want[3]) for x in (ref, got)]
        assert err[0] > 0.0 and err[0] != err[1]
        logs.append(np.log(err[1] / err[0]))
    assert np.exp(np.mean(logs)) < 1.18, np.exp(logs)
