"""The multiscale driver's fused warp, border and error pass: whole solves with
and without the final projection against the same driver with its steps taken
one by one (FLOF_OPT_CFL_SYNC 1: host substep counts, separate advection, border
and error kernels): bit for bit, on extents at and around the least that the
fused pass takes (3), several multisteps, and velocities that need substeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,multi,cfl,width", [
    ((3, 3, 3, 3), 3, 999, 0.1), ((2, 4, 3, 5), 3, 999, 0.1), ((4, 3, 6, 3), 2, 999, -1.0),
    ((24, 21, 23, 17), 3, 999, 0.1), ((24, 21, 23, 17), 4, 999, 0.1), ((24, 21, 23, 17), 1, 999, 0.0),
    ((24, 21, 23, 17), 3, 0.5, 0.1), ((33, 12, 15, 20), 3, 999, 0.4)])
def test_fused_warp_matches_separate_steps(dims, multi, cfl, width):
    import ofblend_gb300 as F
    from ofblend_gb300 import _lib, synth
    ctx = F.Context(0)
    i0 = synth.flow_input(synth.scene_for(0), dims)
    i1 = synth.flow_input(synth.scene_for(1), dims)
    g0 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i0)
    g1 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i1)
    got = []
    for sync in (1, 0):
        ctx.set_option(_lib.FLOF_OPT_CFL_SYNC, sync)
        v = F.Grid4Vec4(dims=dims, ctx=ctx)
        err = F.opticalFlowMultiscale4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-2, postVelBlur=2,
                                        cfl=cfl, multiStep=multi, minGridSize=12, resetBndWidth=width)
        got.append((err, v.to_numpy()))
    assert np.array_equal(got[0][1], got[1][1])
    # the sums over blocks are grouped differently: one float ulp (a border that
    # leaves no cells gives the reference's NaN)
    assert (np.isnan(got[0][0]) and np.isnan(got[1][0])) or abs(got[0][0] - got[1][0]) <= np.spacing(np.float32(abs(got[0][0])))
